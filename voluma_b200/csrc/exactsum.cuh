// Exact, order-independent summation of doubles on the device: the superaccumulator of
// par::ExactSum (src/fvm/parallel/Comm.h:42-93, Comm.cpp:107-164).  Device functions only (no
// kernels), so several translation units can include it.
#pragma once

#include <cuda_runtime.h>

namespace vlm {

// The superaccumulator of par::ExactSum (src/fvm/parallel/Comm.h:42-93, Comm.cpp:107-164):
// a double M*2^E is split over three 32-bit-aligned int64 bins; integer addition is
// associative, so the total does not depend on the summation order, and the final
// conversion reproduces the reference's value bit for bit.
constexpr int kExactBins = 72;
constexpr int kExactStride = kExactBins + 1;  // bins + non-finite flags per partial

// |v| = M 2^(32 i + sh - 1074) over the bins i, i + 1, i + 2, with v's sign (v finite and non-zero).
struct ExactSplit {
    int i;  // -1: nothing to add
    long long lo, mid, hi;
};

__device__ __forceinline__ ExactSplit exact_split(int* flags, double v) {
    ExactSplit t{-1, 0, 0, 0};
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    const int ex = (int)((bits >> 52) & 0x7ff);
    if (ex == 0x7ff) {  // Inf / NaN: remembered as flags (their sum is order independent)
        if ((bits & ((1ull << 52) - 1)) != 0)
            atomicOr(flags, 1);
        else
            atomicOr(flags, (bits >> 63) ? 4 : 2);
        return t;
    }
    long long M = (long long)(bits & ((1ull << 52) - 1));
    if (ex != 0) M |= 1ll << 52;
    if (M == 0) return t;
    const int p = (ex == 0 ? 1 : ex) - 1;
    const int sh = p & 31;
    const long long sgn = -(long long)(bits >> 63);
    t.i = p >> 5;
    t.lo = (M & ((1ll << (32 - sh)) - 1)) << sh;
    const long long r = M >> (32 - sh);
    t.mid = r & 0xFFFFFFFFll;
    t.hi = r >> 32;
    t.lo = (t.lo ^ sgn) - sgn;
    t.mid = (t.mid ^ sgn) - sgn;
    t.hi = (t.hi ^ sgn) - sgn;
    return t;
}

__device__ __forceinline__ void exact_add_split(long long* bins, const ExactSplit& t) {
    atomicAdd((unsigned long long*)&bins[t.i], (unsigned long long)t.lo);
    atomicAdd((unsigned long long*)&bins[t.i + 1], (unsigned long long)t.mid);
    atomicAdd((unsigned long long*)&bins[t.i + 2], (unsigned long long)t.hi);
}

__device__ __forceinline__ void exact_add(long long* bins, int* flags, double v) {
    const ExactSplit t = exact_split(flags, v);
    if (t.i >= 0) exact_add_split(bins, t);
}

// One thread's running sum in the three bins of its latest value.  A warp's values mostly share one
// or two bin positions, so adding each value to shared bins makes 32 lanes queue for the same three
// 64-bit words (each a compare-and-swap loop); the window adds in registers, goes to the bins by
// atomics only when the position changes, and flush_warp() sums what is left of the 32 lanes by
// shuffles, one position at a time.  Integer addition: the totals are the same in any order.
struct ExactWindow {
    ExactSplit w;
    __device__ __forceinline__ void begin() { w = ExactSplit{-1, 0, 0, 0}; }
    __device__ __forceinline__ void add(long long* bins, int* flags, double v) {
        const ExactSplit t = exact_split(flags, v);
        if (t.i < 0) return;
        if (t.i == w.i) {  // each part stays below 2^32 per value: no overflow within 2^31 values
            w.lo += t.lo;
            w.mid += t.mid;
            w.hi += t.hi;
        } else {
            if (w.i >= 0) exact_add_split(bins, w);
            w = t;
        }
    }
    // All 32 lanes; `bins` belongs to this warp alone.
    __device__ __forceinline__ void flush_warp(long long* bins) {
        constexpr unsigned kAll = 0xffffffffu;
        __syncwarp();
        unsigned pending = __ballot_sync(kAll, w.i >= 0);
        while (pending) {
            const int i = __shfl_sync(kAll, w.i, __ffs(pending) - 1);
            const bool mine = w.i == i;
            long long lo = mine ? w.lo : 0, mid = mine ? w.mid : 0, hi = mine ? w.hi : 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                lo += __shfl_down_sync(kAll, lo, o);
                mid += __shfl_down_sync(kAll, mid, o);
                hi += __shfl_down_sync(kAll, hi, o);
            }
            if ((threadIdx.x & 31) == 0) {
                bins[i] += lo;
                bins[i + 1] += mid;
                bins[i + 2] += hi;
            }
            __syncwarp();
            pending &= ~__ballot_sync(kAll, mine);
        }
        w.i = -1;
    }
};

// Carries from bin k0 up to bin k1 (k1's own excess stays in it).
__device__ __forceinline__ void exact_normalize(long long* b, int k0, int k1) {
    for (int k = k0; k < k1; ++k) {
        const long long carry = b[k] >> 32;
        b[k] -= carry * (1ll << 32);
        b[k + 1] += carry;
    }
}

// binsToDouble (Comm.cpp:135-156), on the span of the non-zero bins: a sum's bins are mostly empty,
// and carrying through all of them one after another took longer than adding the partials.  The span
// ends two bins above the highest non-zero one (a bin's carry is below 2^32 in magnitude, so it
// ends in the next bin, and a negative total leaves its sign at the span's top, where the reference
// finds it in its last bin); the digits of |total| are the same on either span.
__device__ inline double exact_value(long long* b, int flags) {
    if (flags & 1) return __longlong_as_double(0x7ff8000000000000ll);
    if ((flags & 6) == 6) return __longlong_as_double(0x7ff8000000000000ll);
    if (flags & 2) return __longlong_as_double(0x7ff0000000000000ll);
    if (flags & 4) return __longlong_as_double((long long)0xfff0000000000000ull);
    int k0 = kExactBins - 1, k1 = 0;
#pragma unroll 8
    for (int k = 0; k < kExactBins; ++k)
        if (b[k] != 0) {
            k0 = min(k0, k);
            k1 = k;
        }
    k1 = min(k1 + 2, kExactBins - 1);
    exact_normalize(b, k0, k1);
    double sign = 1.0;
    if (b[k1] < 0) {
        sign = -1.0;
        for (int k = k0; k <= k1; ++k) b[k] = -b[k];
        exact_normalize(b, k0, k1);
    }
    double r = 0.0;
    for (int k = k1; k >= k0; --k)
        if (b[k] != 0) r += ldexp((double)b[k], 32 * k - 1074);
    return sign * r;
}

}  // namespace vlm
