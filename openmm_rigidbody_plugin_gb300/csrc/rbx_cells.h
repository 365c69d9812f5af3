// rbx_cells.h -- periodic wrapping and list cells of the force field, pure functions shared by the device
// and the host-side tests.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define RBX_HD __host__ __device__
#else
#define RBX_HD
#endif

namespace rbx {

// x wrapped into [0, L): x - L floor(x / L) may round to L itself (x just below zero), or lie an ulp of x
// outside, where the product x / L rounded over an integer; it is then brought back, so that the coordinate
// and its cell always agree. (A coordinate too large to have a place in the box, or a NaN, stays what it is.)
RBX_HD inline float wrap_coordinate(float x, float L, float invL) {
    x = fmaf(-L, floorf(x * invL), x);
    x = x < 0.0f ? x + L : x;
    return x >= L ? x - L : x;
}

// Cell, of nc per edge, of a wrapped coordinate.
RBX_HD inline int cell_of(float x, float invL, int nc) {
    const int c = (int)(x * invL * (float)nc);
    return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

}  // namespace rbx
