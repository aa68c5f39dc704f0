// Host-side construction of the coarse tail's shared-memory images (k_vcycle_tail_parts).
#pragma once

#include <cstdint>
#include <vector>

#include "devtypes.h"
#include "plan.h"

namespace vlm {

struct TailImages {
    std::vector<TailPart> parts;     // `cluster` consecutive parts per system
    std::vector<int32_t> codes;      // value-image gather codes (k_tail_values)
    std::vector<uint16_t> str;       // structure images
    std::vector<int> first;          // per system: the level its tail starts at
    size_t bytes = 0;                // dynamic shared memory of the largest part
};

// Deals every system of `ts` to `cluster` CTAs: each system's tail starts at the first level from
// ts[b].first on whose parts (values of `tsize` bytes) fit `budget` bytes of shared memory a CTA and
// 16-bit local indices.  False when a system's coarsest level alone does not.
bool buildTailImages(const BatchPlan& plan, const std::vector<TailSys>& ts, int cluster, size_t tsize, size_t budget,
                     TailImages& out);

}  // namespace vlm
