// fast_body.cuh -- arithmetic of the fast force mode shared by its kernels
// (k_fast.cu) and the whole-run kernel (k_coop.cuh).
#pragma once
#include <cuda_runtime.h>
#include "femmd_internal.h"
#include "device_common.cuh"

namespace femmd {

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The pair difference on one axis.  IMG: the particle lies within imgD of
// a periodic edge, so an interacting pair may cross it: a difference of
// more than half the box is moved by one box length, rounded once from its
// exact value.
template <bool WRAP, bool IMG>
__device__ __forceinline__ float fdiff(float a, float b, float L) {
    float d = a - b;
    if (WRAP && IMG && fabsf(d) > 0.5f * L) {
        const float sh = d > 0.0f ? L : -L;
        d = (d - sh) + two_sum_err(a, -b, d);
    }
    return d;
}

// x wrapped into [0, L): one box length added or taken away, the reference's
// r - floor(r/L) L for every |r| < 2L (the same single rounding), the full
// expression beyond.
__device__ __forceinline__ float fast_wrap(float x, float L) {
    if (x < 0.0f) x += L;
    else if (x >= L) x -= L;
    if (!(x >= 0.0f && x < L)) x = wrap_coord(x, L);
    return x;
}

}  // namespace femmd
