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
};

// Deals every system of `ts` to `cluster` CTAs: each system's tail starts at the first level from
// ts[b].first on whose parts (values of `tsize` bytes) fit `budget` bytes of shared memory a CTA and
// 16-bit local indices.  first: that level per system; bytes: dynamic shared memory of the largest part.
// False when a system's coarsest level alone does not fit.
bool tailStarts(const BatchPlan& plan, const std::vector<TailSys>& ts, int cluster, size_t tsize, size_t budget,
                std::vector<int>& first, size_t& bytes);

// The images of the systems' levels from first[b] on: the same for both precisions.
bool buildTailImages(const BatchPlan& plan, const std::vector<TailSys>& ts, const std::vector<int>& first, int cluster,
                     TailImages& out);

}  // namespace vlm
