// Starting guesses for point location in a curvilinear vertex grid.
#pragma once

#include <stdint.h>

#include "inside.cuh"

// Element k of an array of n (a debug build's checked read, where one is defined).
#ifndef RG_FLAT_READ
#define RG_FLAT_READ(a, k, n) __ldg((a) + (k))
#endif

namespace rg {

// Approximate cell (ci, cj) of point (px, py) in the grid of nx x ny
// vertices X, Y (row-major): Newton's method on the bilinear index map with
// its analytic Jacobian, in float32.  SINGLE takes the corner-minus-point
// differences from coordinates truncated to float32 (false where they do not
// fit: nothing is set); without it they are taken in float64, so that
// coordinates with a large common offset keep their precision.  It is only a
// starting guess: callers confirm it with the exact containment test and walk
// from it, so its rounding never reaches a result.
template <bool SINGLE>
__device__ __forceinline__ bool seed_cell(const double* __restrict__ X, const double* __restrict__ Y, int64_t nx,
                                          int64_t ny, double px, double py, int64_t* ci, int64_t* cj) {
    const int64_t ncx = nx - 1, ncy = ny - 1;
    float fi = 0.5f * (float)ncx, fj = 0.5f * (float)ncy;
    bool ok = true;
    const float fx = SINGLE ? trunc_float(px, ok) : 0.f, fy = SINGLE ? trunc_float(py, ok) : 0.f;
    auto dx_of = [&](int64_t v) { return SINGLE ? trunc_float(RG_FLAT_READ(X, v, nx * ny), ok) - fx : (float)(RG_FLAT_READ(X, v, nx * ny) - px); };
    auto dy_of = [&](int64_t v) { return SINGLE ? trunc_float(RG_FLAT_READ(Y, v, nx * ny), ok) - fy : (float)(RG_FLAT_READ(Y, v, nx * ny) - py); };
    for (int it = 0; it < 16; it++) {
        int64_t i0 = (int64_t)floorf(fi), j0 = (int64_t)floorf(fj);
        i0 = i0 < 0 ? 0 : (i0 > ncx - 1 ? ncx - 1 : i0);
        j0 = j0 < 0 ? 0 : (j0 > ncy - 1 ? ncy - 1 : j0);
        const float dx = fi - (float)i0, dy = fj - (float)j0;
        const int64_t v00 = i0 * ny + j0, v01 = v00 + 1, v10 = v00 + ny, v11 = v10 + 1;
        const float x00 = dx_of(v00), x01 = dx_of(v01), x10 = dx_of(v10), x11 = dx_of(v11);
        const float y00 = dy_of(v00), y01 = dy_of(v01), y10 = dy_of(v10), y11 = dy_of(v11);
        const float ex = (x00 * (1.f - dy) + x01 * dy) * (1.f - dx) + (x10 * (1.f - dy) + x11 * dy) * dx;
        const float ey = (y00 * (1.f - dy) + y01 * dy) * (1.f - dx) + (y10 * (1.f - dy) + y11 * dy) * dx;
        const float xi = (x10 - x00) * (1.f - dy) + (x11 - x01) * dy;
        const float xj = (x01 - x00) * (1.f - dx) + (x11 - x10) * dx;
        const float yi = (y10 - y00) * (1.f - dy) + (y11 - y01) * dy;
        const float yj = (y01 - y00) * (1.f - dx) + (y11 - y10) * dx;
        const float det = xi * yj - xj * yi;
        if (!(det != 0.f) || !isfinite(det)) break;
        const float di = (yj * ex - xj * ey) / det, dj = (-yi * ex + xi * ey) / det;
        if (!isfinite(di) || !isfinite(dj)) break;
        const float ni = fminf(fmaxf(fi - di, 0.f), (float)ncx), nj = fminf(fmaxf(fj - dj, 0.f), (float)ncy);
        // (SINGLE: a point outside the grid rests at its boundary)
        const bool rest = SINGLE ? fabsf(ni - fi) < 1e-2f && fabsf(nj - fj) < 1e-2f
                                 : fabsf(di) < 1e-2f && fabsf(dj) < 1e-2f;
        fi = ni;
        fj = nj;
        if (rest) break;
    }
    if (!ok) return false;
    int64_t i = (int64_t)floorf(fi), j = (int64_t)floorf(fj);
    *ci = i < 0 ? 0 : (i >= ncx ? ncx - 1 : i);
    *cj = j < 0 ? 0 : (j >= ncy ? ncy - 1 : j);
    return true;
}

// The cell of (px, py) by float32 decisions: 1 inside (*ci, *cj); 0 the walk
// from cell to cell, across the edge the point lies furthest beyond, left the
// grid; -1 not certain which edge that is.  A cell whose containment float32
// leaves open is decided by contains(i, j), in FP64: a few lanes of a warp
// need it, and the seed and walk in FP64, which they took before, are five
// times its operations.  (593 K points in a 1024^2 grid: the walk 72 -> 66 us.)
template <typename Contains>
__device__ __forceinline__ int locate_single(const double* __restrict__ X, const double* __restrict__ Y, int64_t nx,
                                             int64_t ny, double px, double py, int64_t* ci, int64_t* cj,
                                             const Contains& contains) {
    int64_t i, j;
    if (!seed_cell<true>(X, Y, nx, ny, px, py, &i, &j)) return -1;
    for (int step = 0; step < 16; step++) {
        const int64_t v00 = i * ny + j, v10 = v00 + ny;
        const auto at = [&](const double* a, int64_t v) { return RG_FLAT_READ(a, v, nx * ny); };
        const double vx[4] = {at(X, v00), at(X, v10), at(X, v10 + 1), at(X, v00 + 1)};
        const double vy[4] = {at(Y, v00), at(Y, v10), at(Y, v10 + 1), at(Y, v00 + 1)};
        const QuadFilter q(vx, vy, px, py);
        int in = q.contains();
        if (in < 0) in = contains(i, j) ? 1 : 0;
        if (in == 1) {
            *ci = i;
            *cj = j;
            return 1;
        }
        // edge e borders: 0 -> (i, j - 1), 1 -> (i + 1, j), 2 -> (i, j + 1), 3 -> (i - 1, j)
        const int e = q.furthest_edge();
        if (e < 0) return -1;
        i += e == 1 ? 1 : e == 3 ? -1 : 0;
        j += e == 2 ? 1 : e == 0 ? -1 : 0;
        if (i < 0 || j < 0 || i >= nx - 1 || j >= ny - 1) return 0;
    }
    return -1;
}

}  // namespace rg
