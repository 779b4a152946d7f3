// sgd_math.cuh - scalar pieces of the layout updates shared by sgd.cu and
// sgd_small.cu.
#pragma once

#include <cstdint>

#include "common.cuh"

namespace umapb {

__device__ inline float clip4(float v) { return fminf(fmaxf(v, -4.0f), 4.0f); }  // lib.rs:4962

// floor(v).max(0.0) as usize, saturating (lib.rs:5204-5206)
__device__ inline uint32_t floor_count(float v) {
    const float f = floorf(v);
    if (!(f > 0.0f)) return 0u;
    if (f >= 4294967295.0f) return 0xffffffffu;
    return static_cast<uint32_t>(f);
}

// x^y for finite x > 0 through the base-2 logarithm, at a fraction of
// powf's instruction count.  The relative error is about |y log2 x| * 2^-23
// (log2f and exp2f are within 2 ulp): for the exponents used here (b and
// b - 1, |y| <= 2) under 5e-6 at squared distances in [1e-6, 1e6] and under
// 4e-5 anywhere in float range, far below the spread between Hogwild update
// orders.
__device__ __forceinline__ float pow_pos(float x, float y) {
    return exp2f(__fmul_rn(y, log2f(x)));
}

// make_epochs_per_sample (lib.rs:4937-4960) for one edge.
__device__ __forceinline__ float epochs_per_sample(float w, float max_w, float n_epochs_f) {
    const float ns = __fmul_rn(n_epochs_f, __fdiv_rn(w, max_w));
    return ns > 0.0f ? __fdiv_rn(n_epochs_f, ns) : INFINITY;
}

}  // namespace umapb
