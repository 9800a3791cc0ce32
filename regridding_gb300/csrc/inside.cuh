// Float32 images of doubles and the decision of point-in-cell tests by them.
#pragma once

#include <stdint.h>

namespace rg {

// v truncated to float32 from its bits (no FP64 instruction): |v - f| <
// 2^-23 |v|.  Magnitudes below 2^-126 give 0; magnitudes of 2^128 or more (and
// inf, NaN) clear ok.
__device__ __forceinline__ float trunc_float(double v, bool& ok) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned ah = hi & 0x7fffffffu;
    ok = ok && ah < 0x47f00000u;
    const unsigned f = (hi & 0x80000000u) | ((ah - 0x38000000u) << 3) | (lo >> 29);
    return ah < 0x38100000u ? 0.f : __uint_as_float(f);
}

// Whether the extended winding number (regridding/geometry.py:737-829) of a
// quad around a point, as FP64 computes it, is nonzero: 1 inside, 0 outside,
// -1 undecided.  GB300 issues FP64 at 1/64 of its FP32 rate, and the test's
// eight differences, four products and two crossings were most of a locate.
// (593 K points in a 1024^2 grid: the walk kernel 596 us in FP64, 205 us with
// this test, 66 us with the walk itself decided in float32 too.)
//
// With m the largest magnitude of the coordinates and S the largest of the
// eight float32 differences to the point, every difference is within D =
// 2^-21 m + 2^-23 S of the exact one (two truncations of at most 2^-23 of a
// coordinate and one rounding; twice what they add up to).  Where all four y
// differences exceed D their signs are those FP64 computes, and no product of
// two of them (above 2^-126 with S >= 2^-40) vanishes.  The number is then
// the sum over edges whose ends lie on both sides of the point's y of the sign
// of x0 y1 - x1 y0: an edge going up with the point on its left, or down with
// it on its right, counts 1, the others -1, as the upstream's terms do.  The
// float32 cross product is within E = 1.0625 (4 D S + 2 D^2 + 2^-19 S^2) of
// the exact one; where it exceeds E, the crossing's abscissa, |cross| over at
// most 2 S, exceeds 2 D > 2^-22 S, far above the 2^-49 S that FP64 is off by.
struct QuadFilter {
    float x[4], y[4];  // vertices minus the point
    float S, D;        // largest of them, and their error
    bool ok;

    __device__ __forceinline__ QuadFilter(const double* vx, const double* vy, double px, double py) {
        ok = true;
        const float fx = trunc_float(px, ok), fy = trunc_float(py, ok);
        float m = fmaxf(fabsf(fx), fabsf(fy));
        S = 0.f;
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const float a = trunc_float(vx[v], ok), b = trunc_float(vy[v], ok);
            m = fmaxf(m, fmaxf(fabsf(a), fabsf(b)));
            x[v] = __fsub_rn(a, fx);
            y[v] = __fsub_rn(b, fy);
            S = fmaxf(S, fmaxf(fabsf(x[v]), fabsf(y[v])));
        }
        ok = ok && S >= 9.094947e-13f && S <= 1.0995116e12f && m <= 1.0995116e12f;  // 2^-40, 2^40
        D = __fadd_rn(__fmul_rn(4.76837158e-7f, m), __fmul_rn(1.1920929e-7f, S));  // 2^-21 m + 2^-23 S
    }

    __device__ __forceinline__ int contains() const {
        if (!ok) return -1;
        if (!(fminf(fminf(fabsf(y[0]), fabsf(y[1])), fminf(fabsf(y[2]), fabsf(y[3]))) > D)) return -1;
        const float E = __fmul_rn(1.0625f, __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(4.f, D), S), __fmul_rn(__fmul_rn(2.f, D), D)),
                                                     __fmul_rn(__fmul_rn(1.9073486e-6f, S), S)));  // 2^-19
        int w = 0;
        bool sure = true;
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const int p = (v + 3) & 3;
            const float c = __fsub_rn(__fmul_rn(x[p], y[v]), __fmul_rn(x[v], y[p]));
            const bool across = (y[p] < 0.f) != (y[v] < 0.f);
            sure = sure && !(across && !(fabsf(c) > E));
            w += across ? (c > 0.f ? 1 : -1) : 0;
        }
        return sure ? w != 0 : -1;
    }

    // The edge (v -> v + 1) the point lies furthest beyond, 0 to 3, for a
    // quad of either orientation; -1 when that is not clear.
    __device__ __forceinline__ int furthest_edge() const {
        if (!ok) return -1;
        const float turn = (x[0] - x[2]) * (y[1] - y[3]) - (x[1] - x[3]) * (y[0] - y[2]);
        float sc[4], worst = 0.f, second = INFINITY;
        int best = -1;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int f = (e + 1) & 3;
            const float ex = x[f] - x[e], ey = y[f] - y[e];
            const float c = ey * x[e] - ex * y[e];
            sc[e] = (turn < 0.f ? -c : c) * rsqrtf(ex * ex + ey * ey);
            if (sc[e] < worst) {
                second = worst;
                worst = sc[e];
                best = e;
            } else {
                second = fminf(second, sc[e]);
            }
        }
        return best >= 0 && worst < -16.f * D && second - worst > 16.f * D ? best : -1;
    }
};

__device__ __forceinline__ int quad_contains_filter(const double* vx, const double* vy, double px, double py) {
    return QuadFilter(vx, vy, px, py).contains();
}

}  // namespace rg
