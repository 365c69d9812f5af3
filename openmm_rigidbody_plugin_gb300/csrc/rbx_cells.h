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

// Cell, of nc per edge, of a wrapped coordinate (of any other the nearest one, of a NaN the first).
RBX_HD inline int cell_of(float x, float invL, int nc) {
    return (int)fminf(fmaxf(x * invL * (float)nc, 0.0f), (float)(nc - 1));
}

// Cells a to b (none when a > b).
struct CellRange {
    int a, b;
};

// The cells that [x - h, x + h] meets along one edge, `per_length` cells per unit of length, among the w
// cells on either side of cell c, in an unwrapped count (from -w to nc - 1 + w). Any x and h, not finite ones
// too, stay inside that window: the limits are applied before the conversion to whole numbers.
RBX_HD inline CellRange cells_within(float x, float h, float per_length, int c, int w) {
    const float lo = (float)(c - w), hi = (float)(c + w);
    CellRange r;
    r.a = (int)fminf(fmaxf(floorf((x - h) * per_length), lo), hi + 1.0f);
    r.b = (int)fmaxf(fminf(floorf((x + h) * per_length), hi), lo - 1.0f);
    return r;
}

// The part of such a range inside the box (part 0), or across the edge that cell c is near (part 1), as cells
// from 0 to nc - 1. At least 2 w + 1 cells per edge: a range crosses one edge at most.
RBX_HD inline CellRange range_part(CellRange r, int part, int c, int w, int nc) {
    if (part == 0) {
        r.a = r.a > 0 ? r.a : 0;
        r.b = r.b < nc - 1 ? r.b : nc - 1;
    } else if (c < w) {
        r.a += nc;
        r.b = (r.b < -1 ? r.b : -1) + nc;
    } else {
        r.a = (r.a > nc ? r.a : nc) - nc;
        r.b -= nc;
    }
    return r;
}

}  // namespace rbx
