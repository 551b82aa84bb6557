// Bounding boxes as the finder's tests take them (host and device).
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define ATM_HD __host__ __device__ __forceinline__
#else
#define ATM_HD inline
#endif

namespace atm {

// The smaller and the larger of two numbers; no number when either is none, so that a box
// around a box that is no number is none either (fminf and fmaxf would leave that one out).
ATM_HD float bound_min(float a, float b) { return a < b || a != a ? a : b; }
ATM_HD float bound_max(float a, float b) { return a > b || a != a ? a : b; }

// Squared distance between two boxes from the offset of their centres and the sums of their
// half extents.  An axis that is no number counts as no distance: what such a box holds is
// then tested by itself.
ATM_HD float box_gap2(float dx, float dy, float dz, float hx, float hy, float hz) {
    dx = fmaxf(0.f, fabsf(dx) - hx);
    dy = fmaxf(0.f, fabsf(dy) - hy);
    dz = fmaxf(0.f, fabsf(dz) - hz);
    return dx * dx + dy * dy + dz * dz;
}

}  // namespace atm
