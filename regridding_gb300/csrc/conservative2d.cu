// Conservative 2D weights on the GPU: the Ramshaw (1985) edge sweep.
//
// Every grid line of the output grid is traced through the cells of the input
// grid and every grid line of the input grid through the cells of the output
// grid.  Each piece of a line inside one cell of the other grid contributes
// the contour integral 1/2 (x1 y2 - x2 y1) to the two cells of its own grid
// that it separates (Green's theorem); the contributions of one
// (input, output) pair sum to their overlap area.
//
// The walk follows regridding/_weights/_weights_conservative_2d/
// _weights_conservative_2d.py:206-912 step for step with the same IEEE double
// arithmetic (one rounding per operation, no FMA), so crossing decisions,
// emitted triples and their order are identical to the upstream code.  What
// is GB300-specific is the organisation:
//   * seat kernel: one warp per sweep line computes the line's starting state
//     (the O(perimeter) winding-number test is split across the lanes; its
//     partial sums are multiples of 1/2 and therefore exact in any order);
//   * walk: a line is cut into chunks of segments whose starts are guessed; a
//     thread walks a chunk, a warp's lanes stepping together, into slots of the
//     chunk, and a chunk whose start was wrong is walked again.  Slots keep the
//     upstream emission order.  Where they do not fit, one thread per line
//     walks twice (count, then write at scanned offsets);
//   * the O(perimeter) search for re-entry into the static grid
//     (_step_outside_static, :547-698) is answered from a uniform bin grid of
//     the static boundary, evaluating exactly the candidate edges whose
//     bounding boxes can pass the upstream box test and keeping the upstream
//     "first smallest t" choice;
//   * merge: raw triples are bucketed by output cell, a block ranks its rows'
//     triples by (input, emission position) in shared memory, and equal pairs
//     are summed with numpy's add.reduceat association (first + pairwise
//     rest), giving a CSR matrix whose values are bit-identical to the upstream
//     coalesced ones.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "common.cuh"

#ifdef RG_DEBUG
// Debug builds (-DRG_DEBUG, regridding_gb300._build.build(debug=True)): the
// grid reads whose place is computed (seats, guesses, walk) are
// bounds-checked.  A read outside the array sets FLAG_BOUNDS here and yields
// NaN (no trap: the build runs to its end and the host turns the flag into
// RG_ERR_WALK).
namespace rg {
namespace {
__device__ unsigned g_debug_flags;
__device__ __forceinline__ bool debug_in_grid(int64_t i, int64_t j, int64_t nx, int64_t ny) {
    if (i >= 0 && j >= 0 && i < nx && j < ny) return true;
    atomicOr(&g_debug_flags, FLAG_BOUNDS);
    return false;
}
}  // namespace
}  // namespace rg
#define RG_GRID_READ(a, i, j) \
    (debug_in_grid(i, j, nx, ny) ? __ldg((a) + (i) * ny + (j)) : __longlong_as_double(0x7ff8000000000000ll))
#define RG_FLAT_READ(a, k, n) \
    (debug_in_grid(0, k, 1, n) ? __ldg((a) + (k)) : __longlong_as_double(0x7ff8000000000000ll))
#else
#define RG_GRID_READ(a, i, j) __ldg((a) + (i) * ny + (j))
#define RG_FLAT_READ(a, k, n) __ldg((a) + (k))
#endif

#include "inside.cuh"
#include "seed.cuh"

namespace rg {
namespace {

// ---------------------------------------------------------------------------
// geometry (regridding/geometry.py)
// ---------------------------------------------------------------------------

// Order-preserving integer image of a double for the comparisons below:
// keys compare (signed) as the doubles do, -0.0 and +0.0 share a key, and
// NaN is handled by the caller.  Integer compares keep the walk's many
// bounding-box tests off the FP64 pipe (2 lanes per clock per SM on GB300).
__device__ __forceinline__ long long order_key(double v) {
    const long long b = __double_as_longlong(v);
    if ((b & 0x7fffffffffffffffll) == 0) return 0;
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}

__device__ __forceinline__ bool any_nan(double a, double b, double c, double d) {
    const unsigned long long m = 0x7fffffffffffffffull, inf = 0x7ff0000000000000ull;
    return (((unsigned long long)__double_as_longlong(a) & m) > inf) |
           (((unsigned long long)__double_as_longlong(b) & m) > inf) |
           (((unsigned long long)__double_as_longlong(c) & m) > inf) |
           (((unsigned long long)__double_as_longlong(d) & m) > inf);
}

// bounding_boxes_intersect_2d: geometry.py:153-284.  The upstream orders
// each pair and compares min/max; any NaN coordinate makes one of its
// comparisons false, so NaN means no intersection here too.
__device__ __forceinline__ bool bboxes_intersect(double xp1, double yp1, double xp2, double yp2,
                                                 double xq1, double yq1, double xq2, double yq2) {
    if (any_nan(xp1, xp2, xq1, xq2) || any_nan(yp1, yp2, yq1, yq2)) return false;
    long long a = order_key(xp1), b = order_key(xp2), c = order_key(xq1), d = order_key(xq2);
    if (!(min(a, b) <= max(c, d) && min(c, d) <= max(a, b))) return false;
    a = order_key(yp1), b = order_key(yp2), c = order_key(yq1), d = order_key(yq2);
    return min(a, b) <= max(c, d) && min(c, d) <= max(a, b);
}

// two_line_segment_intersection_parameters (geometry.py:370-445) followed by
// two_line_segments_intersect (geometry.py:448-475, half-open 0 <= t,u < 1).
// True only when the rounded quotient fl(n / d) is certainly outside [0, 1),
// decided on the bits without dividing (integer operations; GB300 runs FP64
// at 2 lanes per clock per SM and a division is about ten FP64 operations).
// For |d| < 2^52 (finite):
//   d == 0                  -> n / d is +-inf or NaN;
//   |n| >= |d|              -> |n / d| >= 1, rounds to a magnitude >= 1;
//   n, d of opposite signs  -> n / d < 0, and with |n| >= 2^-1022 its
//                              magnitude exceeds 2^-1075, so it rounds to a
//                              negative number, not to -0.
// Anything else returns false and the caller divides, so the test it
// guards gives the same answer as dividing every time.
__device__ __forceinline__ bool quotient_outside_unit(double n, double d) {
    const unsigned long long abs_mask = 0x7fffffffffffffffull;
    const unsigned long long nb = (unsigned long long)__double_as_longlong(n);
    const unsigned long long db = (unsigned long long)__double_as_longlong(d);
    const unsigned long long na = nb & abs_mask, da = db & abs_mask;
    if (da >= 0x4330000000000000ull) return false;  // |d| >= 2^52, inf or NaN: divide
    if (da == 0 || na >= da) return true;
    return na >= 0x0010000000000000ull && ((nb ^ db) >> 63);
}

// Where the rounded quotient fl(n / d) lies against [0, 1), decided on the
// bits when that is certain: 0 outside, 1 inside, -1 undecided (divide).
// Inside is certain for n == 0, or n and d of one sign with |n| at least two
// representable steps below |d|: then n / d <= 1 - 2^-52, which rounds
// below 1.  Outside follows quotient_outside_unit.  A NaN n is undecided.
__device__ __forceinline__ int quotient_in_unit(double n, double d) {
    const unsigned long long abs_mask = 0x7fffffffffffffffull;
    const unsigned long long nb = (unsigned long long)__double_as_longlong(n);
    const unsigned long long db = (unsigned long long)__double_as_longlong(d);
    const unsigned long long na = nb & abs_mask, da = db & abs_mask;
    if (da >= 0x4330000000000000ull || na > 0x7ff0000000000000ull) return -1;
    if (da == 0 || na >= da) return 0;
    if (na == 0) return 1;
    if ((nb ^ db) >> 63) return na >= 0x0010000000000000ull ? 0 : -1;
    return na + 2 <= da ? 1 : -1;
}

__device__ __forceinline__ bool seg_hit(double x1, double y1, double x2, double y2, double x3,
                                        double y3, double x4, double y4, double* t_out) {
    if (!bboxes_intersect(x1, y1, x2, y2, x3, y3, x4, y4)) return false;
    double tdet = dsub(dmul(dsub(x1, x3), dsub(y3, y4)), dmul(dsub(y1, y3), dsub(x3, x4)));
    double udet = dsub(dmul(dsub(x1, x2), dsub(y1, y3)), dmul(dsub(y1, y2), dsub(x1, x3)));
    double det = dsub(dmul(dsub(x1, x2), dsub(y3, y4)), dmul(dsub(y1, y2), dsub(x3, x4)));
    // most candidate edges miss: reject them before the two divisions
    if (quotient_outside_unit(tdet, det) || quotient_outside_unit(-udet, det)) return false;
    double t = ddiv(tdet, det);
    double u = ddiv(-udet, det);
    *t_out = t;
    return (0 <= t && t < 1) && (0 <= u && u < 1);
}

// ---------------------------------------------------------------------------
// Certified float32 filter for the walk's crossing test.  On GB300 the FP64
// pipe runs 2 lanes per clock per SM (1/64 of FP32), and the 13 FP64
// operations of each candidate edge's determinants were over half of the
// walk.  The filter evaluates the same determinants in float32 from
// coordinates truncated to float32 (from their bits: no FP64 instruction),
// with a static error bound in the manner of Shewchuk's adaptive predicates
// (Shewchuk 1997, "Adaptive precision floating-point arithmetic and fast
// robust geometric predicates"), and answers only where the FP64 result is
// certain; the walk computes the FP64 determinants of the edge it crosses
// (its t is needed) and of the rare undecided candidates.
// ---------------------------------------------------------------------------

// Where q = fl64(n / d) lies against [0, 1), given float32 values nf, df with
// |nf - n| <= E and |df - d| <= E: 1 inside, 0 outside, -1 undecided.
//  * d's sign is certain when |df| > E; with it, nn = nf sgn(d), dn = |df|
//    bound n sgn(d) in [nn - E, nn + E] and |d| in [dn - E, dn + E].
//  * q > 0 when nn - E > 0, and q < 0 when nn + E < 0 (then |q| is far above
//    the smallest double, so it does not round to -0).
//  * q < 1 - 2^-54, which rounds below 1, when (nn + E) / (dn - E) is at most
//    1 - 2^-16 (the two float roundings of the sums move that ratio by a
//    factor of at most (1 + 2^-24) / (1 - 2^-24)); q >= 1, which rounds to
//    at least 1, when nn - E >= (1 + 2^-16)(dn + E).
__device__ __forceinline__ int unit_quotient_filter(float nf, float df, float E) {
    const float dn = fabsf(df);
    if (!(dn > E)) return -1;
    const float nn = df < 0.f ? -nf : nf;
    const float lo = __fsub_rn(nn, E), hi = __fadd_rn(nn, E);
    if (hi < 0.f) return 0;
    if (lo >= __fmul_rn(1.0000152587890625f, __fadd_rn(dn, E))) return 0;
    if (lo > 0.f && hi <= __fmul_rn(0.9999847412109375f, __fsub_rn(dn, E))) return 1;
    return -1;
}

// Float32 decision of the crossing test of the walk's inside step (both
// quotients of seg_hit's determinants in [0, 1)) for segment (x1, y1) ->
// (x1 - dx12, y1 - dy12) and edge (x3, y3) -> (x4, y4), all truncated images
// of the doubles the FP64 test uses, m at least their largest magnitude:
// 1 crossed, 0 not crossed, -1 undecided.
// Error bound: each float difference is within D = 2^-22 m (1 + 2^-21) +
// 2^-24 |diff| (1 + 2^-22) of the FP64 difference (two truncations of at
// most 2^-23 of a coordinate, the float rounding, the FP64 rounding); with
// S the largest float difference, each float determinant is within
// 4 D S + 2 D^2 + 2^-22 S^2 (plus terms of order 2^-53 S^2) of the FP64 one.
// The code takes D = 2^-21 m + 2^-23 S and E = 1.0625 (4 D S + 2 D^2 +
// 2^-19 S^2): twice to eight times those terms, and 6 % for the float
// rounding of E itself.  S is kept in [2^-40, 2^40] (no float underflow or
// overflow in the products); otherwise undecided.
__device__ __forceinline__ int crossing_filter(float x1, float y1, float dx12, float dy12, float x3, float y3,
                                               float x4, float y4, float m) {
    const float x13 = __fsub_rn(x1, x3), y13 = __fsub_rn(y1, y3);
    const float x34 = __fsub_rn(x3, x4), y34 = __fsub_rn(y3, y4);
    const float S = fmaxf(fmaxf(fmaxf(fabsf(x13), fabsf(y13)), fmaxf(fabsf(x34), fabsf(y34))),
                          fmaxf(fabsf(dx12), fabsf(dy12)));
    if (!(S >= 9.094947e-13f && S <= 1.0995116e12f && m <= 1.0995116e12f)) return -1;  // 2^-40, 2^40
    const float T = __fsub_rn(__fmul_rn(x13, y34), __fmul_rn(y13, x34));
    const float U = __fsub_rn(__fmul_rn(dx12, y13), __fmul_rn(dy12, x13));
    const float D = __fsub_rn(__fmul_rn(dx12, y34), __fmul_rn(dy12, x34));
    const float dd = __fadd_rn(__fmul_rn(4.76837158e-7f, m), __fmul_rn(1.1920929e-7f, S));  // 2^-21 m + 2^-23 S
    const float E = __fmul_rn(1.0625f, __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(4.f, dd), S), __fmul_rn(__fmul_rn(2.f, dd), dd)),
                                                 __fmul_rn(__fmul_rn(1.9073486e-6f, S), S)));  // 2^-19
    const int in_t = unit_quotient_filter(T, D, E);
    if (in_t == 0) return 0;
    const int in_u = unit_quotient_filter(-U, D, E);
    if (in_u == 0) return 0;
    return (in_t == 1 && in_u == 1) ? 1 : -1;
}

// -v without the FP64 pipe
__device__ __forceinline__ double negated(double v) {
    return __hiloint2double(__double2hiint(v) ^ INT32_MIN, __double2loint(v));
}

// Whether the rounded quotients tdet / det and udet / det lie in [0, 1), from
// their bits where these decide (almost always).
__device__ __forceinline__ bool in_unit(double tdet, double udet, double det) {
    const int in_t = quotient_in_unit(tdet, det), in_u = quotient_in_unit(udet, det);
    if (in_t == 0 || in_u == 0) return false;
    if (in_t > 0 && in_u > 0) return true;
    const double t = ddiv(tdet, det), u = ddiv(udet, det);
    return (0 <= t && t < 1) && (0 <= u && u < 1);
}

// contribution of one boundary edge to the extended winding number of
// point_is_inside_polygon (geometry.py:737-829)
__device__ __forceinline__ double winding_term(double x, double y, double vx0, double vy0,
                                               double vx1, double vy1) {
    double x0 = dsub(vx0, x), y0 = dsub(vy0, y);
    double x1 = dsub(vx1, x), y1 = dsub(vy1, y);
    if (dmul(y0, y1) < 0) {
        double r = dadd(x0, ddiv(dmul(y0, dsub(x1, x0)), dsub(y0, y1)));
        if (r > 0) return (y0 < 0) ? 1.0 : -1.0;
        return (y0 < 0) ? -1.0 : 1.0;
    } else if (y0 == 0) {
        if (x0 > 0) {
            if (y1 > 0) return 0.5;
            if (y1 < 0) return -0.5;
        } else if (x0 < 0) {
            if (y1 < 0) return 0.5;
            if (y1 > 0) return -0.5;
        }
    } else if (y1 == 0) {
        if (x1 > 0) {
            if (y0 < 0) return 0.5;
            if (y0 > 0) return -0.5;
        } else if (x1 < 0) {
            if (y0 > 0) return 0.5;
            if (y0 < 0) return -0.5;
        }
    }
    return 0.0;
}

struct Grid {
    const double* x;
    const double* y;
    int64_t nx, ny;
    __device__ __forceinline__ double X(int64_t i, int64_t j) const { return RG_GRID_READ(x, i, j); }
    __device__ __forceinline__ double Y(int64_t i, int64_t j) const { return RG_GRID_READ(y, i, j); }
};

// point_is_inside_polygon on the 4 vertices of cell (i, j) in the order
// (i,j), (i+1,j), (i+1,j+1), (i,j+1) (_grids.py:251-276), in float32 where
// that is certain
__device__ bool cell_contains(const Grid& g, int64_t i, int64_t j, double px, double py) {
    double vx[4], vy[4];
    vx[0] = g.X(i, j);         vy[0] = g.Y(i, j);
    vx[1] = g.X(i + 1, j);     vy[1] = g.Y(i + 1, j);
    vx[2] = g.X(i + 1, j + 1); vy[2] = g.Y(i + 1, j + 1);
    vx[3] = g.X(i, j + 1);     vy[3] = g.Y(i, j + 1);
    const int dec = quad_contains_filter(vx, vy, px, py);
    if (dec >= 0) return dec;
    double w = 0;
#pragma unroll
    for (int v = 0; v < 4; v++) {
        int p = (v + 3) & 3;
        w = w + winding_term(px, py, vx[p], vy[p], vx[v], vy[v]);
    }
    return w != 0;
}

// _bilinear_interpolation: regridding/_interp_ndarray.py:226-269
__device__ double bilinear(const double* a, int64_t sx, int64_t sy, double x, double y) {
    int64_t x00 = (int64_t)floor(x), y00 = (int64_t)floor(y);
    if (x00 < 0) x00 = 0;
    else if (x00 > sx - 2) x00 = sx - 2;
    if (y00 < 0) y00 = 0;
    else if (y00 > sy - 2) y00 = sy - 2;
    const int64_t k = x00 * sy + y00, n = sx * sy;
    double a00 = RG_FLAT_READ(a, k, n), a01 = RG_FLAT_READ(a, k + 1, n);
    double a10 = RG_FLAT_READ(a, k + sy, n), a11 = RG_FLAT_READ(a, k + sy + 1, n);
    double dx = dsub(x, (double)x00), dy = dsub(y, (double)y00);
    double w00 = dmul(dsub(1.0, dx), dsub(1.0, dy)), w01 = dmul(dsub(1.0, dx), dy);
    double w10 = dmul(dx, dsub(1.0, dy)), w11 = dmul(dx, dy);
    return dadd(dadd(dadd(dmul(a00, w00), dmul(a01, w01)), dmul(a10, w10)), dmul(a11, w11));
}

__device__ __forceinline__ bool floor_ok(double v) { return isfinite(v) && fabs(v) < 9.0e18; }

// index_of_point_secant: _grids.py:352-463, by one warp (all lanes return the
// same).  Returns false when the upstream falls back to index_of_point_brute
// (singular Jacobian, no convergence, or an iterate the upstream could not
// floor).  An iteration is one chain of dependent FP64 operations, and in one
// lane its six interpolations and the nine cells of the local search were most
// of it: lanes 0 to 5 take one interpolation each and lanes 0 to 8 one cell
// (333 x 257 -> 250 x 193: seats 67 -> 48 us).
__device__ bool locate_secant_warp(const Grid& g, double px, double py, int64_t* oi, int64_t* oj) {
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const double h = 1e-3;
    const int64_t sx = g.nx, sy = g.ny, ncx = sx - 1, ncy = sy - 1;
    // _index_of_point_local (_grids.py:282-349): the first containing cell of
    // the 3 x 3 around (i0, j0), rows first
    auto local = [&](int64_t i0, int64_t j0) {
        const int64_t ii = i0 - 1 + lane / 3, jj = j0 - 1 + lane % 3;
        const bool hit = lane < 9 && ii >= 0 && jj >= 0 && ii < ncx && jj < ncy && cell_contains(g, ii, jj, px, py);
        const unsigned m = __ballot_sync(all, hit);
        const int k = __ffs(m) - 1;
        *oi = m ? i0 - 1 + k / 3 : MAXSIZE;
        *oj = m ? j0 - 1 + k % 3 : MAXSIZE;
    };
    double i = (double)sx / 2, j = (double)sy / 2;
    for (int it = 0; it < 100; it++) {
        // lanes 0, 1: x and y at (i, j); 2, 3: at (i + h, j); 4, 5: at (i, j + h)
        double v = 0.0;
        if (lane < 6)
            v = bilinear(lane & 1 ? g.y : g.x, sx, sy, lane >> 1 == 1 ? dadd(i, h) : i, lane >> 1 == 2 ? dadd(j, h) : j);
        if (!floor_ok(i) || !floor_ok(j)) return false;
        const int64_t i0 = (int64_t)floor(i), j0 = (int64_t)floor(j);
        const double xv = __shfl_sync(all, v, 0), yv = __shfl_sync(all, v, 1);
        const double ex = dsub(xv, px), ey = dsub(yv, py);
        if (i0 >= 0 && j0 >= 0 && i0 < ncx && j0 < ncy) {
            if (cell_contains(g, i0, j0, px, py)) {
                local(i0, j0);
                return true;
            }
        }
        if (fabs(ex) < 1e-10 && fabs(ey) < 1e-10) {
            local(i0, j0);
            return true;
        }
        // lanes 2, 3: dx/di, dy/di; 4, 5: dx/dj, dy/dj
        const double slope = ddiv(dsub(v, lane & 1 ? yv : xv), h);
        const double dx_di = __shfl_sync(all, slope, 2), dy_di = __shfl_sync(all, slope, 3);
        const double dx_dj = __shfl_sync(all, slope, 4), dy_dj = __shfl_sync(all, slope, 5);
        const double det = dsub(dmul(dx_di, dy_dj), dmul(dx_dj, dy_di));
        if (det == 0) return false;
        // lane 0: the step in i, lane 1: in j
        const double a = lane & 1 ? dadd(dmul(-dy_di, ex), dmul(dx_di, ey)) : dsub(dmul(dy_dj, ex), dmul(dx_dj, ey));
        const double step = ddiv(a, det);
        i = dsub(i, __shfl_sync(all, step, 0));
        j = dsub(j, __shfl_sync(all, step, 1));
    }
    return false;
}

// index_of_point_brute (_grids.py:218-279) by one warp: lanes test 32
// consecutive cells of the upstream (i outer, j inner) order per round and
// the first containing cell of the first round with a hit wins.
__device__ void locate_brute_warp(const Grid& g, double px, double py, int64_t* oi, int64_t* oj) {
    int lane = threadIdx.x & 31;
    int64_t ncx = g.nx - 1, ncy = g.ny - 1, ncells = ncx * ncy;
    for (int64_t base = 0; base < ncells; base += 32) {
        int64_t k = base + lane;
        bool hit = k < ncells && cell_contains(g, k / ncy, k % ncy, px, py);
        unsigned m = __ballot_sync(0xffffffffu, hit);
        if (m) {
            int64_t kk = base + __ffs(m) - 1;
            *oi = kk / ncy;
            *oj = kk % ncy;
            return;
        }
    }
    *oi = MAXSIZE;
    *oj = MAXSIZE;
}

// ---------------------------------------------------------------------------
// per-grid preparation
// ---------------------------------------------------------------------------

// grid_volume: _grids.py:50-140.  One thread per cell; the four contour terms
// are added in the upstream order (((0 - A) + B) - C) + D.
__device__ __forceinline__ double cell_area_at(const double* __restrict__ x, const double* __restrict__ y,
                                               int64_t ny, int64_t p, int64_t q) {
    double x00 = x[p * ny + q], y00 = y[p * ny + q];
    double x10 = x[(p + 1) * ny + q], y10 = y[(p + 1) * ny + q];
    double x01 = x[p * ny + q + 1], y01 = y[p * ny + q + 1];
    double x11 = x[(p + 1) * ny + q + 1], y11 = y[(p + 1) * ny + q + 1];
    // axis 0 (transposed, coordinates swapped)
    double A = dmul(dsub(dmul(y00, x10), dmul(y10, x00)), 0.5);
    double B = dmul(dsub(dmul(y01, x11), dmul(y11, x01)), 0.5);
    // axis 1
    double C = dmul(dsub(dmul(x00, y01), dmul(x01, y00)), 0.5);
    double D = dmul(dsub(dmul(x10, y11), dmul(x11, y10)), 0.5);
    double v = dsub(0.0, A);
    v = dadd(v, B);
    v = dsub(v, C);
    v = dadd(v, D);
    return v;
}

__global__ void cell_area_kernel(const double* __restrict__ x, const double* __restrict__ y,
                                 int64_t nx, int64_t ny, double* __restrict__ out) {
    int64_t ncx = nx - 1, ncy = ny - 1;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncx * ncy;
         c += (int64_t)gridDim.x * blockDim.x)
        out[c] = cell_area_at(x, y, ny, c / ncy, c % ncy);
}

// Boundary edges in the scan order of _step_outside_static (:608-683):
// axis 0 (faces i = 0 then i = nx-1, running along j), then axis 1 (faces
// j = 0 then j = ny-1, running along i).
struct Edge {
    double x3, y3, x4, y4;
    int64_t cell;  // flat static cell index
    int code;      // direction_face * 2 + axis = the cell edge it enters through
    int pad;
};

__device__ __forceinline__ Edge boundary_edge(const Grid& g, int64_t k) {
    const int64_t ncx = g.nx - 1, ncy = g.ny - 1;
    int axis, dir;
    int64_t i0, kk = k;
    if (kk < 2 * ncy) {
        axis = 0;
        dir = kk >= ncy;
        i0 = kk - dir * ncy;
    } else {
        kk -= 2 * ncy;
        axis = 1;
        dir = kk >= ncx;
        i0 = kk - dir * ncx;
    }
    Edge e;
    if (axis == 0) {
        int64_t ie = dir ? g.nx - 1 : 0;
        e.x3 = g.X(ie, i0); e.y3 = g.Y(ie, i0);
        e.x4 = g.X(ie, i0 + 1); e.y4 = g.Y(ie, i0 + 1);
        int64_t cx = dir ? ncx - 1 : 0;
        e.cell = cx * ncy + i0;
    } else {
        int64_t je = dir ? g.ny - 1 : 0;
        e.x3 = g.X(i0, je); e.y3 = g.Y(i0, je);
        e.x4 = g.X(i0 + 1, je); e.y4 = g.Y(i0 + 1, je);
        int64_t cy = dir ? ncy - 1 : 0;
        e.cell = i0 * ncy + cy;
    }
    e.code = dir * 2 + axis;
    e.pad = 0;
    return e;
}

struct Bins {
    double ox, oy, inv_h;
    int nbx, nby;
    const int32_t* ptr;    // [nbx*nby + 1] offsets into items
    const int32_t* items;  // edge indices
};

__device__ __forceinline__ int bin_coord(double v, double o, double inv_h, int nb) {
    double f = floor(dmul(dsub(v, o), inv_h));
    if (!(f >= 0)) return 0;  // also maps NaN to 0
    if (f >= nb - 1) return nb - 1;
    return (int)f;
}

// Static-grid preparation of a whole batch.  The static grids are the input
// and the output grid of every pair (grid 2g and 2g + 1 for pair g); they
// share batch-wide arrays, so that every stage below is one launch whatever
// the number of pairs.  Grid k's boundary edges start at edge_base; its
// nbins + 1 bin slots (the last one always empty, so that the grid's slots
// end on its own total) start at bin_base.  Its bins hold offsets into the
// batch's one item array, and its items are edge indices of the grid.
struct PrepGrid {
    Grid g;
    Bins b;
    int64_t cell_base;  // first cell of the pair's input grid in area_in (even k only)
    int64_t edge_base;
    int64_t bin_base;
};

// grid k whose edges hold batch edge e (edge bases rise strictly: a grid has
// at least four boundary edges)
__device__ __forceinline__ int grid_of_edge(const PrepGrid* __restrict__ P, int n, int64_t e) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P[mid].edge_base <= e) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Areas of the input cells of every pair, in area_in's order (pair by pair),
// each with its reciprocal for area_ratio.
__device__ __forceinline__ void cell_areas(unsigned block, const PrepGrid* __restrict__ P, int G, int64_t ncells,
                                           double2* __restrict__ out) {
    const int64_t c = block * (int64_t)blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    int lo = 0, hi = G - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P[2 * mid].cell_base <= c) lo = mid;
        else hi = mid - 1;
    }
    const Grid g = P[2 * lo].g;
    const int64_t local = c - P[2 * lo].cell_base, ncy = g.ny - 1;
    const double a = cell_area_at(g.x, g.y, g.ny, local / ncy, local % ncy);
    out[c] = make_double2(a, ddiv(1.0, a));
}

// a / cell.x, correctly rounded, from the cell's rounded reciprocal cell.y:
// two corrections by the exact remainder.  The product a * y is within 1.5
// units of the quotient; the first correction leaves at most half a unit and
// 2^-53 of one, and the second then rounds as the quotient does (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000", 1990: the
// remainder is exact, and its product with y's error stays below the distance
// of any quotient from a rounding boundary).  Operands outside 2^-400 .. 2^400,
// where nothing here over- or underflows, zeros and NaN divide.  (Half the
// FP64 operations of a division.  2048^2 -> 1536^2: with the loads of both sides
// issued together the scattering pass takes 0.79 ms in place of 0.93, the
// areas 0.20 in place of 0.16.)
__device__ __forceinline__ bool ratio_range(double v) {
    return ((unsigned)__double2hiint(v) >> 20 & 0x7ffu) - 623u <= 800u;
}
__device__ __forceinline__ double area_ratio(double a, double2 cell) {
    if (!(ratio_range(a) && ratio_range(cell.x))) return ddiv(a, cell.x);
    const double q0 = dmul(a, cell.y);
    const double q1 = __fma_rn(__fma_rn(-cell.x, q0, a), cell.y, q0);
    return __fma_rn(__fma_rn(-cell.x, q1, a), cell.y, q1);
}

// Bounding boxes (xmin, ymin, xmax, ymax) of every static grid: nparts
// blocks of 256 threads per grid fold strided vertices into partial
// extrema, then one warp per grid combines them (min and max are exact in
// any order, so the partition does not matter).
__device__ __forceinline__ void box_parts(unsigned block, const PrepGrid* __restrict__ P, int nparts,
                                          double* __restrict__ part) {
    __shared__ long long sh[4][8];
    const int k = block / nparts, p = block % nparts;
    const Grid g = P[k].g;
    const int64_t n = g.nx * g.ny;
    // extrema of the order keys (no FP64 instruction); NaN is left out, and
    // no vertex gives the infinities
    long long a = order_key(INFINITY), b = a, c = order_key(-INFINITY), d = c;
    for (int64_t v = (int64_t)p * blockDim.x + threadIdx.x; v < n; v += (int64_t)nparts * blockDim.x) {
        const double xv = g.x[v], yv = g.y[v];
        if (!any_nan(xv, xv, xv, xv)) {
            a = min(a, order_key(xv));
            c = max(c, order_key(xv));
        }
        if (!any_nan(yv, yv, yv, yv)) {
            b = min(b, order_key(yv));
            d = max(d, order_key(yv));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = min(b, __shfl_xor_sync(0xffffffffu, b, o));
        c = max(c, __shfl_xor_sync(0xffffffffu, c, o));
        d = max(d, __shfl_xor_sync(0xffffffffu, d, o));
    }
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        sh[0][warp] = a;
        sh[1][warp] = b;
        sh[2][warp] = c;
        sh[3][warp] = d;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        long long r = sh[threadIdx.x][0];
        for (int w = 1; w < 8; w++) r = threadIdx.x < 2 ? min(r, sh[threadIdx.x][w]) : max(r, sh[threadIdx.x][w]);
        // the key's double: the keys' map is its own inverse
        part[((int64_t)k * nparts + p) * 4 + threadIdx.x] =
            __longlong_as_double(r ^ ((r >> 63) & 0x7fffffffffffffffll));
    }
}

__global__ void bbox_combine_batch(const double* __restrict__ part, int nparts, int ngrids, double* __restrict__ out) {
    const int k = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (k >= ngrids) return;  // whole warps leave together
    const double* q = part + (int64_t)k * nparts * 4;
    double a = INFINITY, b = INFINITY, c = -INFINITY, d = -INFINITY;
    for (int i = lane; i < nparts; i += 32) {
        a = fmin(a, q[4 * i]);
        b = fmin(b, q[4 * i + 1]);
        c = fmax(c, q[4 * i + 2]);
        d = fmax(d, q[4 * i + 3]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a = fmin(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = fmin(b, __shfl_xor_sync(0xffffffffu, b, o));
        c = fmax(c, __shfl_xor_sync(0xffffffffu, c, o));
        d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
    }
    if (lane == 0) {
        out[4 * k] = a;
        out[4 * k + 1] = b;
        out[4 * k + 2] = c;
        out[4 * k + 3] = d;
    }
}

// What the builds of a batch prepare from the vertices alone, by one launch of
// 256 threads a block: the first box_blocks blocks the parts of the bounding
// boxes, edge_blocks the boundary edges, the rest the input cells' areas.
__global__ void __launch_bounds__(256)
    prepare_batch(const PrepGrid* __restrict__ P, int G, unsigned box_blocks, int nparts, double* __restrict__ part,
                  unsigned edge_blocks, int64_t nedges, Edge* __restrict__ edges, int64_t ncells,
                  double2* __restrict__ areas) {
    if (blockIdx.x < box_blocks) {
        box_parts(blockIdx.x, P, nparts, part);
    } else if (blockIdx.x < box_blocks + edge_blocks) {
        const int64_t e = (blockIdx.x - box_blocks) * (int64_t)blockDim.x + threadIdx.x;
        if (e >= nedges) return;
        const int k = grid_of_edge(P, 2 * G, e);
        edges[e] = boundary_edge(P[k].g, e - P[k].edge_base);
    } else {
        cell_areas(blockIdx.x - box_blocks - edge_blocks, P, G, ncells, areas);
    }
}

// Every edge goes to each bin its bounding box touches: a counting pass,
// then (after the scan of the counts) a filing pass.  The order of the
// items within a bin depends on the atomics; the outside step that reads
// them is order-independent.
template <bool FILL>
__global__ void bin_edges_batch(const PrepGrid* __restrict__ P, int ngrids, const Edge* __restrict__ edges,
                                int64_t nedges, unsigned* __restrict__ counts, int32_t* __restrict__ items,
                                const int64_t* __restrict__ ptr64) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nedges;
         k += (int64_t)gridDim.x * blockDim.x) {
        const int gk = grid_of_edge(P, ngrids, k);
        const Bins b = P[gk].b;
        const int64_t base = P[gk].bin_base;
        const Edge e = edges[k];
        int bx0 = bin_coord(fmin(e.x3, e.x4), b.ox, b.inv_h, b.nbx);
        int bx1 = bin_coord(fmax(e.x3, e.x4), b.ox, b.inv_h, b.nbx);
        int by0 = bin_coord(fmin(e.y3, e.y4), b.oy, b.inv_h, b.nby);
        int by1 = bin_coord(fmax(e.y3, e.y4), b.oy, b.inv_h, b.nby);
        for (int by = by0; by <= by1; by++)
            for (int bx = bx0; bx <= bx1; bx++) {
                const int64_t bin = base + (int64_t)by * b.nbx + bx;
                unsigned pos = atomicAdd(&counts[bin], 1u);
                if (FILL) items[ptr64[bin] + pos] = (int32_t)(k - P[gk].edge_base);
            }
    }
}

__global__ void i64_to_i32(const int64_t* a, int32_t* b, int64_t n) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x)
        b[k] = (int32_t)a[k];
}

// ---------------------------------------------------------------------------
// sweep families and line seats
// ---------------------------------------------------------------------------

struct Static {
    Grid g;
    int64_t ncx, ncy;
    double blx, bly, bux, buy;
    int64_t nbound;  // boundary polygon vertices
    const Edge* edges;
    Bins bins;
};

struct Family {
    Grid sweep;        // unaligned sweep grid
    int transposed;    // axis_sweep == 0
    int64_t lines;     // aligned rows
    int64_t len;       // aligned columns (vertices along a line)
    int sweep_input;
    int axis;
    int st;            // 0: static = input grid, 1: static = output grid
    int64_t line_base;
    __device__ __forceinline__ double SX(int64_t a, int64_t b) const {
        return transposed ? sweep.X(b, a) : sweep.X(a, b);
    }
    __device__ __forceinline__ double SY(int64_t a, int64_t b) const {
        return transposed ? sweep.Y(b, a) : sweep.Y(a, b);
    }
};

struct SweepParams {
    Family fam[4];
    Static st[2];
    const double2* area_in;  // (ncx_in, ncy_in): area and its reciprocal
    const double* w_in;     // nullable
    int64_t ncy_in, ncy_out;
    int64_t total_lines;
};

struct Seat {
    int64_t stx, sty;
    int outside;
    int pad;
};

__device__ __forceinline__ int family_of(const SweepParams& P, int64_t line) {
    int f = 0;
#pragma unroll
    for (int k = 1; k < 4; k++)
        if (line >= P.fam[k].line_base) f = k;
    return f;
}

// A batch of grid pairs swept together: per pair its sweep parameters and
// chunk plan (whose line, chunk and slot bases are global across the batch),
// prefix bases of its lines, chunks and output rows, and its own error word.
// Kernels find their pair by binary search over the prefix bases.
struct ChunkPlan;
struct Batch {
    const SweepParams* P;    // [G]
    const ChunkPlan* C;      // [G] (null for whole-line walks)
    const int64_t* line_base;   // [G + 1]
    const int64_t* chunk_base;  // [G + 1]
    const int64_t* out_base;    // [G + 1] first output row of every pair
    unsigned* flags;            // [G]
    int G;
};

// the pair owning global index x: the largest g with base[g] <= x
__device__ __forceinline__ int pair_of(const int64_t* __restrict__ base, int G, int64_t x) {
    int lo = 0, hi = G - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= x) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Starting state of a sweep line (:439-468), by one warp.
__device__ void seat_line(const Batch& B, int64_t line, Seat* seats) {
    const int lane = threadIdx.x & 31;
    const int pg = pair_of(B.line_base, B.G, line);
    const SweepParams& P = B.P[pg];
    unsigned* flags = B.flags + pg;
    const Family& F = P.fam[family_of(P, line)];
    const Static& S = P.st[F.st];
    int64_t li = line - F.line_base;
    double x1 = F.SX(li, 0), y1 = F.SY(li, 0);
    Seat seat;
    seat.stx = MAXSIZE;
    seat.sty = MAXSIZE;
    seat.outside = 1;
    seat.pad = 0;
    bool in_box = (S.blx <= x1 && x1 <= S.bux) && (S.bly <= y1 && y1 <= S.buy);
    if (in_box) {
        // Winding number of the boundary polygon at the line's first vertex.
        // Only edges whose y-range holds y1 have a nonzero term, and all of
        // them lie in the row of edge bins at y1's bin (bin_coord is
        // monotone); an edge spanning several x-bins of the row is counted
        // in its first.  The boundary edges run along the polygon's order on
        // the faces j = 0 and i = nx - 1 and against it on i = 0 and
        // j = ny - 1 (codes 0 and 3), where their ends are swapped back.
        // The terms are 0, +-1/2 and +-1, so the sum is exact in any order.
        double w = 0;
        const Bins& BN = S.bins;
        const int row = bin_coord(y1, BN.oy, BN.inv_h, BN.nby);
        for (int bx = lane; bx < BN.nbx; bx += 32) {
            const int64_t bin = (int64_t)row * BN.nbx + bx;
            const int32_t q0 = __ldg(BN.ptr + bin), q1 = __ldg(BN.ptr + bin + 1);
            for (int32_t q = q0; q < q1; q++) {
                const Edge e = S.edges[__ldg(BN.items + q)];
                if (bin_coord(fmin(e.x3, e.x4), BN.ox, BN.inv_h, BN.nbx) != bx) continue;
                if (e.code == 0 || e.code == 3) w += winding_term(x1, y1, e.x4, e.y4, e.x3, e.y3);
                else w += winding_term(x1, y1, e.x3, e.y3, e.x4, e.y4);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (w != 0) {
            int64_t i = MAXSIZE, j = MAXSIZE;
            if (!locate_secant_warp(S.g, x1, y1, &i, &j)) locate_brute_warp(S.g, x1, y1, &i, &j);
            if (i == MAXSIZE) {
                // the upstream would index out of range here; report it and
                // leave the line outside so the walk stays in bounds
                if (lane == 0) atomicOr(flags, FLAG_SEAT_OUTSIDE);
            } else {
                seat.stx = i;
                seat.sty = j;
                seat.outside = 0;
            }
        }
    }
    if (lane == 0) seats[line] = seat;
}

__global__ void __launch_bounds__(128) seat_kernel(Batch B, Seat* seats) {
    const int64_t line = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (line < B.line_base[B.G]) seat_line(B, line, seats);
}

// ---------------------------------------------------------------------------
// the walk
// ---------------------------------------------------------------------------

// State of a walk at a sweep vertex.  At every vertex the upstream's
// entry-edge marker is back at sys.maxsize and the current point is the
// vertex itself, so (outside, static cell) is the whole state.
struct WalkState {
    int64_t stx, sty;
    int64_t sy;  // index of the sweep vertex the walk is at
    int outside;
    int pad;
};

// The bins of the static boundary that the box (x0, x1) x (y0, y1) of a
// segment's float32 images may touch, one or two more than FP64 would give:
// every candidate is tested against the segment itself, so more bins change
// nothing.  False: certainly none (the box lies beside the boundary's).
// *bx1 < 0: float32 cannot tell, FP64 has to.  An image is within 2^-23 of its
// coordinate (at most m) or 2^-126; e is four times what two of them and the
// roundings add up to.  (The box and bins in FP64 were a fifth of the walk's
// FP64 operations on 2048^2 -> 1536^2.)
__device__ __forceinline__ bool boundary_bins(const Static& S, bool ok, float x0, float x1, float y0, float y1, float m,
                                              int* bx0, int* bx1, int* by0, int* by1) {
    const float lx = trunc_float(S.blx, ok), ux = trunc_float(S.bux, ok);
    const float ly = trunc_float(S.bly, ok), uy = trunc_float(S.buy, ok);
    const Bins& B = S.bins;
    const float ox = trunc_float(B.ox, ok), oy = trunc_float(B.oy, ok), inv = trunc_float(B.inv_h, ok);
    m = fmaxf(m, fmaxf(fmaxf(fmaxf(fabsf(lx), fabsf(ux)), fmaxf(fabsf(ly), fabsf(uy))), fmaxf(fabsf(ox), fabsf(oy))));
    *bx1 = -1;
    ok = ok && m <= 1.0995116e12f;                                          // 2^40
    const float e = __fadd_rn(__fmul_rn(9.53674316e-7f, m), 1.17549435e-36f);  // 2^-20 m + 100 * 2^-126
    if (!ok) return true;
    if (x1 + e < lx || x0 - e > ux || y1 + e < ly || y0 - e > uy) return false;
    const float nx = (float)(B.nbx - 1), ny = (float)(B.nby - 1);
    const float w = __fadd_rn(__fmul_rn(e, inv), __fmul_rn(9.53674316e-7f, fmaxf(nx, ny)));
    if (!(w < 0.5f)) return true;
    *bx0 = (int)fminf(fmaxf((x0 - ox) * inv - w, 0.f), nx);
    *bx1 = (int)fminf(fmaxf((x1 - ox) * inv + w, 0.f), nx);
    *by0 = (int)fminf(fmaxf((y0 - oy) * inv - w, 0.f), ny);
    *by1 = (int)fminf(fmaxf((y1 - oy) * inv + w, 0.f), ny);
    return true;
}

// The body of the prange loop of _sweep_along_axis (:432-533) with
// _step_outside_static (:547-698), _step_inside_static (:707-895) and
// _calc_and_save_weights (:903-976) inlined, run on line li from vertex
// st.sy until the walk reaches vertex j_end.  EMIT_TRIPLES stores (input cell,
// output cell, weight) for each of the line's sides at [wpos, wend),
// EMIT_PIECES one (static cell, sweep segment, area) for both; past wend they
// only count (and flag the overflow), as EMIT_COUNT does throughout.  Returns
// the number of triples or pieces.
//
// The lanes of a warp in `lanes` call it together and step together, those
// that have ended too: left to themselves they leave the loop over a cell's
// edges at different turns and stay apart (8.6 of 32 lanes in the FP64 part of
// a step, which costs the same for one lane as for 32).  2048^2 -> 1536^2: the
// walk 3.73 ms, with lanes together 2.74, with two searches per crossing and
// open edges decided beside it 2.34, with 32-bit state and float32 boundary
// bins 2.12.  (96 registers for 10 blocks per SM in place of 8: 2.04 ms, but
// builds of 333x257 and less are 2 % slower.)
constexpr int EMIT_COUNT = 0, EMIT_TRIPLES = 1, EMIT_PIECES = 2;
template <int EMIT>
__device__ int64_t walk_range(const SweepParams& P, const Family& F, const Static& S, int64_t li, int64_t j_end,
                              WalkState& state, int64_t wpos, int64_t wend, int32_t* __restrict__ raw_in,
                              int32_t* __restrict__ raw_out, double* __restrict__ raw_val, unsigned* flags,
                              int64_t max_steps, unsigned lanes) {
    // 32-bit indices: cells and vertices are counted below 2^31 and 2^32
    const double* __restrict__ const vx = S.g.x;
    const double* __restrict__ const vy = S.g.y;
    const unsigned row = (unsigned)S.g.ny;  // vertices from one to the next along the first axis
    const int ncx = (int)S.ncx, ncy = (int)S.ncy;
    const auto vertex = [&](int x, int y, int v) {  // indices_cell_vertex: _grids.py:153-158
#ifdef RG_DEBUG
        if (!debug_in_grid(x + ((v + 1) >> 1 & 1), y + (v >> 1), S.g.nx, S.g.ny)) return 0u;
#endif
        return (unsigned)x * row + (unsigned)y + ((v + 1) >> 1 & 1 ? row : 0u) + (unsigned)(v >> 1);
    };
    const int64_t along = F.transposed ? F.sweep.ny : 1;  // from one vertex of the line to the next
    const double* __restrict__ const lx = F.sweep.x + (F.transposed ? li : li * F.sweep.ny);
    const double* __restrict__ const ly = F.sweep.y + (F.transposed ? li : li * F.sweep.ny);
    const auto line_vertex = [&](const double* __restrict__ line, int k) {
#ifdef RG_DEBUG
        if (!debug_in_grid(F.transposed ? k : li, F.transposed ? li : k, F.sweep.nx, F.sweep.ny))
            return __longlong_as_double(0x7ff8000000000000ll);
#endif
        return __ldg(line + k * along);
    };
    bool outside = state.outside;
    int stx = outside ? 0 : (int)state.stx, sty = outside ? 0 : (int)state.sty;
    constexpr int NONE = -1;
    int edge_last = NONE;
    int sy_idx = (int)state.sy, end = (int)j_end;
    int n_emit = 0;
    int steps = 0;
    const int step_limit = (int)(max_steps < INT32_MAX ? max_steps : INT32_MAX);
    double x1 = line_vertex(lx, sy_idx), y1 = line_vertex(ly, sy_idx);
    int first = 0;  // the edge that the search in a cell begins with

    // the piece of the current segment from (x1, y1) to (xe, ye)
    const auto emit = [&](double xe, double ye) {
        // _calc_and_save_weights: area_triangle, negated for axis 0
        double area = dmul(dsub(dmul(x1, ye), dmul(xe, y1)), 0.5);
        if (F.axis == 0) area = negated(area);
        // when the static grid is the input grid both sides share the
        // input cell, and -area / a_in (times w_in) is exactly the
        // negation of area / a_in (times w_in): one division serves both
        double w_static = 0.0;
        bool have_static = false;
        if constexpr (EMIT == EMIT_PIECES) {
            if (wpos < wend) {
                raw_in[wpos] = stx * ncy + sty;
                raw_out[wpos] = sy_idx;
                raw_val[wpos] = area;
            } else {
                atomicOr(flags, FLAG_CAPACITY);
            }
            wpos++;
            n_emit++;
        } else {
#pragma unroll
            for (int side = 0; side < 2; side++) {
                int64_t is = side == 0 ? li - 1 : li;
                if (side == 0 && !(is >= 0)) continue;
                if (side == 1 && !(is < F.lines - 1)) continue;
                int64_t a = is, b = sy_idx;
                if (F.axis == 0) { a = sy_idx; b = is; }
                int64_t ii, ij, oi, oj;
                if (F.sweep_input) { ii = a; ij = b; oi = stx; oj = sty; }
                else { ii = stx; ij = sty; oi = a; oj = b; }
                int64_t in_flat = ii * P.ncy_in + ij;
                if constexpr (EMIT == EMIT_TRIPLES) {
                    if (wpos < wend) {
                        double w;
                        if (!F.sweep_input && have_static) {
                            w = -w_static;
                        } else {
                            w = area_ratio(side == 0 ? area : -area, __ldg(P.area_in + in_flat));
                            if (P.w_in) w = dmul(w, __ldg(P.w_in + in_flat));
                            if (!F.sweep_input && side == 0) {
                                w_static = w;
                                have_static = true;
                            }
                        }
                        raw_in[wpos] = (int32_t)in_flat;
                        raw_out[wpos] = (int32_t)(oi * P.ncy_out + oj);
                        raw_val[wpos] = w;
                    } else {
                        // never write past the slots given to this walk
                        atomicOr(flags, FLAG_CAPACITY);
                    }
                    wpos++;
                }
                n_emit++;
            }
        }
    };

    while (true) {
        const bool live = sy_idx < end;
        if (!__any_sync(lanes, live)) break;
        bool inside = false;
        double x2 = x1, y2 = y1;
        bool enter = false;
        if (live && steps >= step_limit) {
            atomicOr(flags, FLAG_WALK_CAP);
            end = sy_idx;
        } else if (live) {
            x2 = line_vertex(lx, sy_idx + 1);
            y2 = line_vertex(ly, sy_idx + 1);
            inside = !outside;
            enter = outside;
        }
        if (enter) {
            // _step_outside_static: smallest-t crossing of the static boundary,
            // candidates from the bins overlapping the segment's box
            const double p2x = x2, p2y = y2;
            bool found = false;
            double t_min = INFINITY;
            // float32 images of the segment for the crossing filter
            bool seg_ok = true;
            const float x1f = trunc_float(x1, seg_ok), y1f = trunc_float(y1, seg_ok);
            const float x2f = trunc_float(p2x, seg_ok), y2f = trunc_float(p2y, seg_ok);
            const float dx12f = __fsub_rn(x1f, x2f), dy12f = __fsub_rn(y1f, y2f);
            const float mseg = fmaxf(fmaxf(fabsf(x1f), fabsf(y1f)), fmaxf(fabsf(x2f), fabsf(y2f)));
            int best_order = INT32_MAX, best_code = 0, best_cell = 0;
            const Bins& B = S.bins;
            int bx0, bx1, by0, by1;
            if (boundary_bins(S, seg_ok, fminf(x1f, x2f), fmaxf(x1f, x2f), fminf(y1f, y2f), fmaxf(y1f, y2f), mseg, &bx0,
                              &bx1, &by0, &by1)) {
                if (bx1 < 0) {
                    bx0 = bin_coord(fmin(x1, p2x), B.ox, B.inv_h, B.nbx);
                    bx1 = bin_coord(fmax(x1, p2x), B.ox, B.inv_h, B.nbx);
                    by0 = bin_coord(fmin(y1, p2y), B.oy, B.inv_h, B.nby);
                    by1 = bin_coord(fmax(y1, p2y), B.oy, B.inv_h, B.nby);
                }
                for (int by = by0; by <= by1; by++) {
                    for (int bx = bx0; bx <= bx1; bx++) {
                        int64_t bin = (int64_t)by * B.nbx + bx;
                        int32_t s0 = __ldg(B.ptr + bin), s1 = __ldg(B.ptr + bin + 1);
                        for (int32_t q = s0; q < s1; q++) {
                            int32_t ek = __ldg(B.items + q);
                            const Edge e = S.edges[ek];
                            if (!bboxes_intersect(x1, y1, p2x, p2y, e.x3, e.y3, e.x4, e.y4)) continue;
                            {
                                // most candidate boundary edges are certainly not crossed
                                bool ok = seg_ok;
                                const float x3f = trunc_float(e.x3, ok), y3f = trunc_float(e.y3, ok);
                                const float x4f = trunc_float(e.x4, ok), y4f = trunc_float(e.y4, ok);
                                const float m = fmaxf(mseg, fmaxf(fmaxf(fabsf(x3f), fabsf(y3f)),
                                                                  fmaxf(fabsf(x4f), fabsf(y4f))));
                                if (ok && crossing_filter(x1f, y1f, dx12f, dy12f, x3f, y3f, x4f, y4f, m) == 0) continue;
                            }
                            double t;
                            if (!seg_hit(x1, y1, p2x, p2y, e.x3, e.y3, e.x4, e.y4, &t)) continue;
                            if ((int)e.cell == edge_last) continue;
                            if (t < t_min || (t == t_min && ek < best_order)) {
                                t_min = t;
                                best_order = ek;
                                best_code = e.code;
                                best_cell = (int)e.cell;
                                found = true;
                            }
                        }
                    }
                }
            }
            if (found) {
                stx = best_cell / ncy;
                sty = best_cell % ncy;
                x2 = dadd(x1, dmul(t_min, dsub(p2x, x1)));
                y2 = dadd(y1, dmul(t_min, dsub(p2y, y1)));
                edge_last = best_code;
                outside = false;
            } else {
                edge_last = NONE;
                sy_idx = sy_idx + 1;
            }
            steps++;
        }
        __syncwarp(lanes);
        // _step_inside_static: first crossed edge of the current static cell
        // other than the entry edge.  The hit test of each candidate edge is
        // seg_hit's, decided in float32 where that is certain; an edge that is
        // left open ends the search and is decided with its crossing below,
        // where the FP64 operations of both are the same.  A lane whose
        // segment ends in its cell writes that piece and searches with the
        // next segment, so that most lanes come to the crossing with one to
        // compute: an FP64 instruction costs the same for one lane as for 32.
        // Same edges, same order, same t.
        int found = -1;
        bool open = false;
        bool look = inside;
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) {
            if (look) {
                // float32 images of the segment for the crossing filter
                bool seg_ok = true;
                const float x1f = trunc_float(x1, seg_ok), y1f = trunc_float(y1, seg_ok);
                const float x2f = trunc_float(x2, seg_ok), y2f = trunc_float(y2, seg_ok);
                const float dx12f = __fsub_rn(x1f, x2f), dy12f = __fsub_rn(y1f, y2f);
                const float mseg = fmaxf(fmaxf(fabsf(x1f), fabsf(y1f)), fmaxf(fabsf(x2f), fabsf(y2f)));
                bool ok3 = seg_ok;
                const unsigned k3 = vertex(stx, sty, 3);
                float x3f = trunc_float(__ldg(vx + k3), ok3), y3f = trunc_float(__ldg(vy + k3), ok3);
#pragma unroll 1
                for (int v = 0; v < 4; v++) {
                    const unsigned k4 = vertex(stx, sty, v);
                    bool ok4 = seg_ok;
                    const float x4f = trunc_float(__ldg(vx + k4), ok4), y4f = trunc_float(__ldg(vy + k4), ok4);
                    if (found < 0 && v >= first && v != edge_last) {
                        // 1: crossed, 0: not crossed (both certain), -1: open.
                        // (A certain crossing is one of the boxes, too.)
                        int dec = -1;
                        const float m =
                            fmaxf(mseg, fmaxf(fmaxf(fabsf(x3f), fabsf(y3f)), fmaxf(fabsf(x4f), fabsf(y4f))));
                        if (ok3 && ok4) dec = crossing_filter(x1f, y1f, dx12f, dy12f, x3f, y3f, x4f, y4f, m);
                        if (dec != 0) found = v;
                        open = dec < 0;
                    }
                    x3f = x4f;
                    y3f = y4f;
                    ok3 = ok4;
                }
            }
            __syncwarp(lanes);
            if (pass == 1) break;
            look = look && found < 0;
            if (look) {
                emit(x2, y2);
                steps++;
                edge_last = NONE;
                first = 0;
                x1 = x2;
                y1 = y2;
                look = inside = ++sy_idx < end;
                if (inside) {
                    x2 = line_vertex(lx, sy_idx + 1);
                    y2 = line_vertex(ly, sy_idx + 1);
                }
            }
            __syncwarp(lanes);
        }
        if (found >= 0) {
            const unsigned k3 = vertex(stx, sty, (found + 3) & 3), k4 = vertex(stx, sty, found);
            const double x3 = __ldg(vx + k3), y3 = __ldg(vy + k3), x4 = __ldg(vx + k4), y4 = __ldg(vy + k4);
            const double dx12 = dsub(x1, x2), dy12 = dsub(y1, y2);
            const double x13 = dsub(x1, x3), y13 = dsub(y1, y3);
            const double x34 = dsub(x3, x4), y34 = dsub(y3, y4);
            const double tdet = dsub(dmul(x13, y34), dmul(y13, x34));
            const double det = dsub(dmul(dx12, y34), dmul(dy12, x34));
            if (open) {
                open = !bboxes_intersect(x1, y1, x2, y2, x3, y3, x4, y4) ||
                       !in_unit(tdet, negated(dsub(dmul(dx12, y13), dmul(dy12, x13))), det);
            }
            if (!open) {
                // x1 + t (x2 - x1), with x2 - x1 the negated difference at hand
                const double t = ddiv(tdet, det);
                x2 = dsub(x1, dmul(t, dx12));
                y2 = dsub(y1, dmul(t, dy12));
            }
        }
        __syncwarp(lanes);
        if (open) {
            // not crossed after all: on with the next edge
            first = found + 1;
            continue;
        }
        if (inside) {
            emit(x2, y2);
            steps++;
            first = 0;
            const int cell = stx * ncy + sty;
            if (found >= 0) {
                stx += found & 1 ? 0 : found - 1;  // cell_normals: _grids.py:143-148
                sty += found & 1 ? found - 2 : 0;
                edge_last = (found + 2) & 3;
            } else {
                sy_idx++;
                edge_last = NONE;
            }
            if (!(stx >= 0 && sty >= 0 && stx < ncx && sty < ncy)) {
                edge_last = cell;
                outside = true;
            }
        }
        x1 = x2;  // (unchanged where the walk has ended)
        y1 = y2;
    }
    state.stx = outside ? MAXSIZE : stx;
    state.sty = outside ? MAXSIZE : sty;
    state.sy = sy_idx;
    state.outside = outside;
    return n_emit;
}

// One thread per sweep line over the whole line.  COUNT mode only counts the
// triples a line emits; WRITE mode stores them from offsets[line].
template <bool WRITE>
__global__ void __launch_bounds__(64)
    walk_kernel(Batch B, const Seat* __restrict__ seats, int64_t* __restrict__ counts,
                const int64_t* __restrict__ offsets, int32_t* __restrict__ raw_in,
                int32_t* __restrict__ raw_out, double* __restrict__ raw_val) {
    int64_t line = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const unsigned here = __ballot_sync(0xffffffffu, line < B.line_base[B.G]);
    if (line >= B.line_base[B.G]) return;
    const int pg = pair_of(B.line_base, B.G, line);
    const SweepParams& P = B.P[pg];
    const Family F = P.fam[family_of(P, line)];
    const Static& S = P.st[F.st];
    Seat seat = seats[line];
    WalkState state{seat.stx, seat.sty, 0, seat.outside, 0};
    const int64_t max_steps = 64 * (F.len + 4 * (S.ncx + S.ncy) + 16);
    int64_t n = walk_range<WRITE ? EMIT_TRIPLES : EMIT_COUNT>(P, F, S, line - F.line_base, F.len - 1, state,
                                  WRITE ? offsets[line] : 0, WRITE ? offsets[line + 1] : 0, raw_in, raw_out,
                                  raw_val, B.flags + pg, max_steps, here);
    if (!WRITE) counts[line] = n;
    if (WRITE && B.out_base[pg] != 0) {
        // output rows of the batch: the pair's rows follow those of the pairs before it
        const int32_t ob = (int32_t)B.out_base[pg];
        for (int64_t q = offsets[line]; q < offsets[line] + n; q++) raw_out[q] += ob;
    }
}

// ---------------------------------------------------------------------------
// chunked walk: every line is cut into chunks of CH sweep segments that are
// walked in parallel.  A chunk starts from its vertex located in the static
// grid; a per-line repair pass then re-walks, in order, every chunk whose
// start disagrees with the end state of the chunk before it, so the pieces
// are exactly those of one sequential walk per line.  A piece stands for the
// triples of both cells that its line separates; their weights are divided
// out where the triples are ordered, a piece per lane, and not in the walk,
// whose FP64 instructions run with half their lanes (2048^2 -> 1536^2: walk
// 4.71 -> 3.86 ms, the two ordering passes 1.38 -> 1.62 ms then).
// ---------------------------------------------------------------------------

struct ChunkPlan {
    int64_t ch;              // sweep segments per chunk
    int64_t nc[4];           // chunks per line, per family
    int64_t chunk_base[5];   // first chunk id of each family (and the total)
    int64_t cap[4];          // piece slots per chunk, per family
    int64_t slot_base[4];    // first slot of each family
};

__device__ __forceinline__ int family_of_chunk(const ChunkPlan& C, int64_t g) {
    int f = 0;
#pragma unroll
    for (int k = 1; k < 4; k++)
        if (g >= C.chunk_base[k]) f = k;
    return f;
}

// A guess of the walk state at a sweep vertex: the static cell containing
// it (Newton seed on the bilinear index map, then a walk across the edge the
// point lies beyond), or "outside".  Wrong guesses are fixed by the repair.
__device__ WalkState guess_state(const Static& S, double px, double py, int64_t sy) {
    WalkState w{MAXSIZE, MAXSIZE, sy, 1, 0};
    if (!((S.blx <= px && px <= S.bux) && (S.bly <= py && py <= S.buy))) return w;
    const Grid& g = S.g;
    const int64_t ncx = S.ncx, ncy = S.ncy;
    int64_t ci, cj;
    const int single = locate_single(g.x, g.y, g.nx, g.ny, px, py, &ci, &cj,
                                     [&](int64_t i, int64_t j) { return cell_contains(g, i, j, px, py); });
    if (single == 1) return WalkState{ci, cj, sy, 0, 0};
    if (single == 0) return w;
    seed_cell<false>(g.x, g.y, g.nx, g.ny, px, py, &ci, &cj);
    for (int step = 0; step < 64; step++) {
        if (cell_contains(g, ci, cj, px, py)) {
            w.stx = ci;
            w.sty = cj;
            w.outside = 0;
            return w;
        }
        double vx[4] = {g.X(ci, cj), g.X(ci + 1, cj), g.X(ci + 1, cj + 1), g.X(ci, cj + 1)};
        double vy[4] = {g.Y(ci, cj), g.Y(ci + 1, cj), g.Y(ci + 1, cj + 1), g.Y(ci, cj + 1)};
        double area2 = (vx[0] - vx[2]) * (vy[1] - vy[3]) - (vx[1] - vx[3]) * (vy[0] - vy[2]);
        double sgn = area2 >= 0 ? 1.0 : -1.0;
        int best = -1;
        double worst = 0;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            int f = (e + 1) & 3;
            double ex = vx[f] - vx[e], ey = vy[f] - vy[e];
            double cr = sgn * (ex * (py - vy[e]) - ey * (px - vx[e]));
            double len = sqrt(ex * ex + ey * ey);
            double sc = len > 0 ? cr / len : 0;
            if (sc < worst) {
                worst = sc;
                best = e;
            }
        }
        if (best < 0) break;
        const int di[4] = {0, 1, 0, -1};
        const int dj[4] = {-1, 0, 1, 0};
        int64_t ni = ci + di[best], nj = cj + dj[best];
        if (ni < 0 || nj < 0 || ni >= ncx || nj >= ncy) break;
        ci = ni;
        cj = nj;
    }
    return w;
}

// Starts of all chunks: the first blocks seat the lines, a warp each, for the
// lines' first chunks; the others guess, a thread for each further chunk.  Both
// are chains of dependent steps on few threads, so they run side by side.
__global__ void __launch_bounds__(128)
    chunk_seat_kernel(Batch B, unsigned seat_blocks, Seat* __restrict__ seats, WalkState* __restrict__ starts,
                      int64_t* __restrict__ counts) {
    if (blockIdx.x < seat_blocks) {
        const int64_t line = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
        if (line >= B.line_base[B.G]) return;
        seat_line(B, line, seats);
        if ((threadIdx.x & 31) == 0) {
            const int pg = pair_of(B.line_base, B.G, line);
            const SweepParams& P = B.P[pg];
            const ChunkPlan& C = B.C[pg];
            const int f = family_of(P, line);
            const Seat s0 = seats[line];
            starts[C.chunk_base[f] + (line - P.fam[f].line_base) * C.nc[f]] = WalkState{s0.stx, s0.sty, 0, s0.outside, 0};
        }
        return;
    }
    int64_t g = (blockIdx.x - seat_blocks) * (int64_t)blockDim.x + threadIdx.x;
    if (g >= B.chunk_base[B.G]) {
        if (g == B.chunk_base[B.G]) counts[g] = 0;  // the scan's last element
        return;
    }
    const int pg = pair_of(B.chunk_base, B.G, g);
    const SweepParams& P = B.P[pg];
    const ChunkPlan& C = B.C[pg];
    int f = family_of_chunk(C, g);
    const Family& F = P.fam[f];
    int64_t k = g - C.chunk_base[f];
    int64_t li = k / C.nc[f], c = k - li * C.nc[f];
    int64_t j0 = c * C.ch;
    if (c > 0) starts[g] = guess_state(P.st[F.st], F.SX(li, j0), F.SY(li, j0), j0);
}

__device__ __forceinline__ int64_t chunk_end(const ChunkPlan& C, const Family& F, int64_t c) {
    int64_t e = (c + 1) * C.ch;
    return e < F.len - 1 ? e : F.len - 1;
}

__device__ __forceinline__ void chunk_walk_one(const Batch& B, const WalkState* __restrict__ starts,
                                               WalkState* __restrict__ ends, int64_t* __restrict__ counts,
                                               int32_t* __restrict__ s_in, int32_t* __restrict__ s_out,
                                               double* __restrict__ s_val, int64_t g, unsigned lanes) {
    const int pg = pair_of(B.chunk_base, B.G, g);
    const SweepParams& P = B.P[pg];
    const ChunkPlan& C = B.C[pg];
    unsigned* flags = B.flags + pg;
    int f = family_of_chunk(C, g);
    const Family F = P.fam[f];
    const Static& S = P.st[F.st];
    int64_t k = g - C.chunk_base[f];
    int64_t li = k / C.nc[f], c = k - li * C.nc[f];
    WalkState st = starts[g];
    int64_t base = C.slot_base[f] + k * C.cap[f];
    const int64_t max_steps = 64 * (C.ch + 4 * (S.ncx + S.ncy) + 16);
    counts[g] = walk_range<EMIT_PIECES>(P, F, S, li, chunk_end(C, F, c), st, base, base + C.cap[f], s_in, s_out,
                                 s_val, flags, max_steps, lanes);
    ends[g] = st;
}

// Every warp walks the 32 chunks of its own number, then takes 32 more from a
// counter.  Its lanes step together (walk_range): lanes that finish early wait,
// which costs less than the divergence did when every lane took its next chunk
// by itself (2048^2 -> 1536^2: 2.1 ms, 3.7 ms before; FP64 issue takes 55 % of
// it, the latency of the steps the rest).
__global__ void __launch_bounds__(64)
    chunk_walk_kernel(Batch B, const WalkState* __restrict__ starts, WalkState* __restrict__ ends,
                      int64_t* __restrict__ counts, int32_t* __restrict__ s_in, int32_t* __restrict__ s_out,
                      double* __restrict__ s_val, unsigned long long* __restrict__ next_chunk) {
    const int64_t total = B.chunk_base[B.G];
    const int64_t threads = (int64_t)gridDim.x * blockDim.x;
    int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const unsigned lane = threadIdx.x & 31u;
    while (true) {
        const unsigned here = __ballot_sync(0xffffffffu, g < total);
        if (here == 0) return;
        if (g < total) chunk_walk_one(B, starts, ends, counts, s_in, s_out, s_val, g, here);
        __syncwarp();
        if (total <= threads) return;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(next_chunk, 32ull);
        base = __shfl_sync(0xffffffffu, base, 0);
        g = threads + (int64_t)base + lane;
    }
}

// One warp per line: chunks are walked again, in order, wherever a chunk's
// start differs from the previous chunk's end.  The lanes compare 32 chunks at
// a time; a chunk walked again changes its own end, so the comparison goes on
// from the chunk after it.  (A thread per line compared its chunks one dependent
// load after another: 69 us for the 84 chunks a line of 333 x 257 -> 250 x 193,
// now 4 us.)
__global__ void __launch_bounds__(128)
    chunk_repair_kernel(Batch B, WalkState* __restrict__ starts, WalkState* __restrict__ ends,
                        int64_t* __restrict__ counts, int32_t* __restrict__ s_in, int32_t* __restrict__ s_out,
                        double* __restrict__ s_val, unsigned long long* __restrict__ n_repaired) {
    const int lane = threadIdx.x & 31;
    const int64_t line = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (line >= B.line_base[B.G]) return;  // whole warps
    const int pg = pair_of(B.line_base, B.G, line);
    const SweepParams& P = B.P[pg];
    const ChunkPlan& C = B.C[pg];
    unsigned* flags = B.flags + pg;
    int f = family_of(P, line);
    const Family& F = P.fam[f];
    const Static& S = P.st[F.st];
    int64_t li = line - F.line_base;
    const int64_t max_steps = 64 * (C.ch + 4 * (S.ncx + S.ncy) + 16);
    int64_t g0 = C.chunk_base[f] + li * C.nc[f];
    for (int64_t c0 = 1; c0 < C.nc[f];) {
        bool same = true;
        if (c0 + lane < C.nc[f]) {
            const WalkState prev = ends[g0 + c0 + lane - 1], cur = starts[g0 + c0 + lane];
            same = prev.outside == cur.outside && (prev.outside || (prev.stx == cur.stx && prev.sty == cur.sty));
        }
        const unsigned differ = __ballot_sync(0xffffffffu, !same);
        if (!differ) {
            c0 += 32;
            continue;
        }
        // A walk of the pair has met its step cap: its weights are an error, and
        // a line that cycles would do so in each of its chunks again.
        unsigned fl = 0;
        if (lane == 0) fl = *(const volatile unsigned*)flags;
        if (__shfl_sync(0xffffffffu, fl, 0) & FLAG_WALK_CAP) return;
        const int64_t c = c0 + __ffs(differ) - 1;
        if (lane == 0) {
            atomicAdd(n_repaired, 1ull);
            const WalkState prev = ends[g0 + c - 1];
            starts[g0 + c] = prev;
            WalkState st = prev;
            int64_t k = li * C.nc[f] + c;
            int64_t base = C.slot_base[f] + k * C.cap[f];
            counts[g0 + c] = walk_range<EMIT_PIECES>(P, F, S, li, chunk_end(C, F, c), st, base, base + C.cap[f], s_in,
                                              s_out, s_val, flags, max_steps, 1u);
            ends[g0 + c] = st;
        }
        __syncwarp();
        c0 = c + 1;
    }
}

// ---------------------------------------------------------------------------
// merge (regridding/_weights/_weights_arrays.py:44-73)
// ---------------------------------------------------------------------------

// ---------------------------------------------------------------------------
// Output-row ordering of the chunked walk's triples, made from the pieces in
// the chunks' slots (no compacted copy, no index indirection): piece q of
// chunk g has raw positions 2 (offsets[g] + q) and the next one for its two
// triples (the order of one sequential walk per line), and each goes to the
// bucket of its output row with the key (input cell << 32 | raw position), so
// that ordering each row by key gives the same order as the bucket sort of the
// compacted triples: by input cell, then by raw position.  In the counting and
// scattering passes LANES lanes of a warp take a chunk, a piece per lane (a
// chunk's consecutive triples often share a row, and their lanes add to its
// counter once); 8 or 16 where chunks hold few pieces.  The counting pass keeps
// every triple's place in its bucket, so the scattering one needs no atomics
// (2048^2 -> 1536^2: counting 0.22 -> 0.26 ms, scattering 1.07 -> 0.93 ms).  order_rows
// sorts and merges the buckets.
// ---------------------------------------------------------------------------

// What a chunk's pieces share, and the cells of its piece's two triples
// (_calc_and_save_weights, :903-976): side 0 lies below the line, side 1 above.
struct PieceLine {
    const SweepParams* P;
    const Family* F;
    int64_t li;
    __device__ __forceinline__ bool has(int side) const { return side == 0 ? li >= 1 : li < F->lines - 1; }
    __device__ __forceinline__ void cells(int side, int32_t stat, int32_t seg, int32_t* in, int32_t* out) const {
        const int64_t is = side == 0 ? li - 1 : li;
        const int64_t a = F->axis == 0 ? seg : is, b = F->axis == 0 ? is : seg;
        const int32_t own = (int32_t)(a * (F->sweep_input ? P->ncy_in : P->ncy_out) + b);
        *in = F->sweep_input ? own : stat;
        *out = F->sweep_input ? stat : own;
    }
};

// the chunk's line, and its first slot
__device__ __forceinline__ PieceLine piece_line(const Batch& B, int pg, int64_t g, int64_t* base) {
    const ChunkPlan& C = B.C[pg];
    const int f = family_of_chunk(C, g);
    const int64_t k = g - C.chunk_base[f];
    *base = C.slot_base[f] + k * C.cap[f];
    return PieceLine{&B.P[pg], &B.P[pg].fam[f], k / C.nc[f]};
}

__device__ __forceinline__ unsigned warp_row_add(unsigned* counters, int32_t b, bool active) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned key = active ? (unsigned)b : 0xffffffffu;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const unsigned leader = __ffs(peers) - 1;
    unsigned base = 0;
    if (active && lane == leader) base = atomicAdd(&counters[b], (unsigned)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + __popc(peers & ((1u << lane) - 1u));
}

// A triple in its row's bucket: one 16-byte store (key and weight in arrays of
// their own touched two sectors per triple: 2048^2 -> 1536^2 1.37 ms, now 1.07).
struct __align__(16) Triple {
    int64_t key;  // input cell << 32 | raw position
    double w;
};

template <int LANES>
__global__ void slot_count_rows(Batch B, const int64_t* __restrict__ counts, const int32_t* __restrict__ s_cell,
                                const int32_t* __restrict__ s_seg, unsigned* __restrict__ rows,
                                uint2* __restrict__ s_pos) {
    const int lane = threadIdx.x & (LANES - 1);
    const int64_t total = B.chunk_base[B.G];
    int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES;
    const bool valid = g < total;
    if (!__any_sync(0xffffffffu, valid)) return;
    if (!valid) g = total - 1;
    const int pg = pair_of(B.chunk_base, B.G, g);
    int64_t base;
    const PieceLine L = piece_line(B, pg, g, &base);
    const int32_t ob = (int32_t)B.out_base[pg];
    const int64_t n = valid ? counts[g] : 0;
    for (int64_t q = lane; __any_sync(0xffffffffu, q < n); q += LANES) {
        const bool active = q < n;
        const int32_t cell = active ? s_cell[base + q] : 0, seg = active ? s_seg[base + q] : 0;
        unsigned pos[2];
#pragma unroll
        for (int side = 0; side < 2; side++) {
            int32_t in, out;
            L.cells(side, cell, seg, &in, &out);
            pos[side] = warp_row_add(rows, active ? out + ob : 0, active && L.has(side));
        }
        if (active) s_pos[base + q] = make_uint2(pos[0], pos[1]);
    }
}

template <int LANES>
__global__ void __launch_bounds__(256)
    slot_scatter_rows(Batch B, const int64_t* __restrict__ counts, const int64_t* __restrict__ offsets,
                                  const int32_t* __restrict__ s_cell, const int32_t* __restrict__ s_seg,
                                  const double* __restrict__ s_area, const uint2* __restrict__ s_pos,
                                  const int64_t* __restrict__ row_start, Triple* __restrict__ triples) {
    const int lane = threadIdx.x & (LANES - 1);
    const int64_t total = B.chunk_base[B.G];
    const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES;
    if (g >= total) return;
    const int pg = pair_of(B.chunk_base, B.G, g);
    int64_t base;
    const PieceLine L = piece_line(B, pg, g, &base);
    const int32_t ob = (int32_t)B.out_base[pg];
    const int n = (int)counts[g];
    const unsigned order0 = 2 * (unsigned)offsets[g];
    // the moving grid's cell beside segment seg is seg * step + own0 before the line, + own1 after it
    const bool has0 = L.has(0), has1 = L.has(1), sweep_input = L.F->sweep_input;
    const int32_t nc = (int32_t)(sweep_input ? L.P->ncy_in : L.P->ncy_out);
    const int32_t step = L.F->axis == 0 ? nc : 1, other = L.F->axis == 0 ? 1 : nc;
    const int32_t own1 = (int32_t)L.li * other, own0 = own1 - other;
    const double2* __restrict__ area_in = L.P->area_in;
    const double* __restrict__ w_in = L.P->w_in;
    row_start += ob;
    s_cell += base;
    s_seg += base;
    s_area += base;
    s_pos += base;
    for (int q = lane; q < n; q += LANES) {
        const int32_t cell = s_cell[q], seg = s_seg[q] * step;
        const double area = s_area[q];
        const uint2 pos = s_pos[q];
        const int32_t c0 = seg + own0, c1 = seg + own1;
        const int64_t to0 = has0 ? row_start[sweep_input ? cell : c0] + pos.x : 0;
        const int64_t to1 = has1 ? row_start[sweep_input ? cell : c1] + pos.y : 0;
        const int32_t in0 = sweep_input ? (has0 ? c0 : c1) : cell, in1 = sweep_input && has1 ? c1 : in0;
        // a static input grid: both sides share the input cell, and
        // -area / a_in (times w_in) is exactly the negation of area / a_in
        // (times w_in): one division serves both
        const double2 a0 = __ldg(area_in + in0);
        double w0 = area_ratio(area, a0);
        if (w_in) w0 = dmul(w0, __ldg(w_in + in0));
        double w1 = negated(w0);
        if (sweep_input) {
            w1 = negated(area_ratio(area, __ldg(area_in + in1)));
            if (w_in) w1 = dmul(w1, __ldg(w_in + in1));
        }
        if (has0) triples[to0] = Triple{(int64_t)in0 << 32 | (order0 + 2 * q), w0};
        if (has1) triples[to1] = Triple{(int64_t)in1 << 32 | (order0 + 2 * q + 1), w1};
    }
}

__global__ void make_keys(const int32_t* raw_in, int64_t n, int64_t* skey) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x)
        skey[k] = ((int64_t)raw_in[k] << 32) | (int64_t)(uint32_t)k;
}

// numpy's pairwise summation for n <= 128 (used by add.reduce / reduceat):
// a sequential sum from -0.0 below 8 terms, else 8 interleaved partial sums.
template <typename At>
__device__ double pw_block(const At& at, int64_t off, int64_t n) {
    if (n < 8) {
        double res = -0.0;
        for (int64_t i = 0; i < n; i++) res = dadd(res, at(off + i));
        return res;
    }
    double r[8];
#pragma unroll
    for (int j = 0; j < 8; j++) r[j] = at(off + j);
    int64_t i = 8;
    for (; i < n - (n % 8); i += 8) {
#pragma unroll
        for (int j = 0; j < 8; j++) r[j] = dadd(r[j], at(off + i + j));
    }
    double res = dadd(dadd(dadd(r[0], r[1]), dadd(r[2], r[3])), dadd(dadd(r[4], r[5]), dadd(r[6], r[7])));
    for (; i < n; i++) res = dadd(res, at(off + i));
    return res;
}

// numpy pairwise_sum: blocks of at most 128 terms, larger ranges split at
// n/2 rounded down to a multiple of 8 (iterative form of the recursion)
template <typename At>
__device__ double pairwise_sum(const At& at, int64_t off, int64_t n) {
    struct Frame {
        int64_t off, n;
        double left;
        int stage;
    };
    Frame stk[48];
    int sp = 0;
    stk[0] = {off, n, 0.0, 0};
    for (;;) {
        Frame& f = stk[sp];
        if (f.n <= 128) {
            double result = pw_block(at, f.off, f.n);
            for (;;) {
                if (sp == 0) return result;
                sp--;
                Frame& p = stk[sp];
                if (p.stage == 1) {
                    p.left = result;
                    p.stage = 2;
                    int64_t n2 = p.n / 2;
                    n2 -= n2 % 8;
                    stk[sp + 1] = {p.off + n2, p.n - n2, 0.0, 0};
                    sp++;
                    break;
                }
                result = dadd(p.left, result);
            }
        } else {
            f.stage = 1;
            int64_t n2 = f.n / 2;
            n2 -= n2 % 8;
            stk[sp + 1] = {f.off, n2, 0.0, 0};
            sp++;
        }
    }
}


// The sum of the run [g, h), by the add.reduceat association (a run of up to
// 129 is one block of the pairwise sum).
template <typename At>
__device__ __forceinline__ double run_sum(const At& at, int64_t g, int64_t h) {
    return dadd(at(g), h - g - 1 <= 128 ? pw_block(at, g + 1, h - g - 1) : pairwise_sum(at, g + 1, h - g - 1));
}

// Merges the entries [s, t) of a row, sorted by input cell, by run_sum; the
// reads and stores (in place) are the caller's.  Returns the end of the merged
// entries.
template <typename In, typename At, typename Store>
__device__ __forceinline__ int64_t merge_sorted(int64_t s, int64_t t, const In& in, const At& at, const Store& store) {
    int64_t w = s, g = s;
    while (g < t) {
        const int32_t c = in(g);
        int64_t h = g + 1;
        while (h < t && in(h) == c) h++;
        store(w, c, run_sum(at, g, h));
        w++;
        g = h;
    }
    return w;
}

// Buckets to merged rows, `per` rows per block, a thread per triple, then
// one per merged entry.  The keys go to shared memory; a triple's rank is the
// number of keys of its row below its own (keys are unique); it is stored at
// its rank, the first of a row marked.  Each run of one input cell is then
// added up and written, without gaps from the block's first bucket's start.
// Blocks with a row of more than ROW_SMALL or rows of more than BLOCK_TRIPLES
// triples are listed for order_rows_long.  (2048^2 -> 1536^2, 22 triples per
// row: 0.75 ms, and 0.07 ms for copy_blocks; bound by instructions, half of
// them the ranking.  A warp per row in the ranking and a lane per row in the
// merge took 0.98 ms; a launch each for ranking, merging and compacting
// through global memory 0.78, 0.42 and 0.17 ms.)
// The host takes 32, 8 or 2 rows per block, for up to 40, 160 or more triples
// per row, so that a block's rows mostly fit BLOCK_TRIPLES (2048^2 -> 300^2,
// 230 triples per row: with 32 every block was listed and order_rows_long took
// 10.2 ms; now 1.5.)
constexpr int ORDER_ROWS = 32;  // at most
__host__ __forceinline__ int order_rows_per_block(int64_t triples, int64_t rows) {
    return triples <= 40 * rows ? 32 : triples <= 160 * rows ? 8 : 2;
}
constexpr int ORDER_THREADS = 256;
constexpr int ROW_SMALL = 1024;      // a row's ranks cost its square
constexpr int BLOCK_TRIPLES = 2048;  // 40 KB of shared memory
constexpr int32_t ROW_HEAD = INT32_MIN;

// Rows' merged counts to their prefix (pre[ORDER_ROWS] the total); by one warp.
__device__ __forceinline__ void order_counts(int mine, int* pre) {
    const int lane = threadIdx.x & 31;
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += up;
    }
    pre[lane + 1] = incl;
    if (lane == 0) pre[0] = 0;
}

template <int PER>
__global__ void __launch_bounds__(ORDER_THREADS)
    order_rows(const int64_t* __restrict__ row_start, int64_t nrows, const Triple* __restrict__ triples,
               int32_t* __restrict__ tmp_col, double* __restrict__ tmp_val, int64_t* __restrict__ row_nnz,
               int2* __restrict__ long_list, unsigned* __restrict__ long_count) {
    __shared__ int64_t key[BLOCK_TRIPLES];
    __shared__ double val[BLOCK_TRIPLES];
    __shared__ int32_t in[BLOCK_TRIPLES];
    __shared__ int start[PER + 1];
    __shared__ unsigned heads[BLOCK_TRIPLES / 32 + 1];  // a bit per triple that begins a run
    __shared__ int before[BLOCK_TRIPLES / 32 + 1];      // runs before each word of heads
    const int t = threadIdx.x, lane = t & 31;
    const int64_t r0 = (int64_t)blockIdx.x * PER, s0 = row_start[r0];
    bool longer = false;
    if (t == 0 && blockIdx.x == 0) row_nnz[nrows] = 0;  // the scan's last element
    if (t <= PER) {
        const int64_t r = r0 + t < nrows ? r0 + t : nrows, s = row_start[r];
        longer = t == PER ? s - s0 > BLOCK_TRIPLES : r < nrows && row_start[r + 1] - s > ROW_SMALL;
        start[t] = (int)(s - s0);
    }
    if (__syncthreads_or(longer)) {
        if (t == 0) long_list[atomicAdd(long_count, 1u)] = make_int2((int)blockIdx.x, 0);
        return;
    }
    const int n = start[PER];
    for (int e = t; e < n; e += ORDER_THREADS) key[e] = triples[s0 + e].key;
    __syncthreads();
    for (int e = t; e < n; e += ORDER_THREADS) {
        int r = 0;
#pragma unroll
        for (int d = PER / 2; d > 0; d >>= 1)
            if (start[r + d] <= e) r += d;
        const int s = start[r], m = start[r + 1];
        const int64_t mine = key[e];
        int rank = 0;
#pragma unroll 4
        for (int j = s; j < m; j++) rank += key[j] < mine;
        in[s + rank] = (int32_t)(mine >> 32) | (rank == 0 ? ROW_HEAD : 0);
        val[s + rank] = triples[s0 + e].w;
    }
    __syncthreads();
    const int words = n / 32 + 1;
    for (int q = t >> 5; q < words; q += ORDER_THREADS / 32) {
        const int e = q * 32 + lane;
        const bool head = e < n && (in[e] < 0 || in[e] != (in[e - 1] & ~ROW_HEAD));
        const unsigned word = __ballot_sync(0xffffffffu, head);
        if (lane == 0) heads[q] = word;
    }
    __syncthreads();
    if (t < 32) {
        int sum = 0;
        for (int q0 = 0; q0 < words; q0 += 32) {
            int incl = q0 + lane < words ? __popc(heads[q0 + lane]) : 0;
            const int own = incl;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += up;
            }
            if (q0 + lane < words) before[q0 + lane] = sum + incl - own;
            sum += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    const auto runs_before = [&](int e) { return before[e >> 5] + __popc(heads[e >> 5] & ((1u << (e & 31)) - 1u)); };
    if (t < PER && r0 + t < nrows) row_nnz[r0 + t] = runs_before(start[t + 1]) - runs_before(start[t]);
    uint16_t* run = reinterpret_cast<uint16_t*>(key);  // where each run begins
    for (int e = t; e < n; e += ORDER_THREADS)
        if (heads[e >> 5] >> (e & 31) & 1u) run[runs_before(e)] = (uint16_t)e;
    const int runs = runs_before(n);
    if (t == 0) run[runs] = (uint16_t)n;
    __syncthreads();
    for (int k = t; k < runs; k += ORDER_THREADS) {
        const int g = run[k];
        tmp_col[s0 + k] = in[g] & ~ROW_HEAD;
        tmp_val[s0 + k] = run_sum([&](int64_t e) { return val[e]; }, g, run[k + 1]);
    }
}

// A row of up to ROW_SHORT triples ranked and merged by a warp, through its
// triples' place; returns its merged entries.
constexpr int ROW_SHORT = 256;
__device__ int order_short_row(int64_t s, int len, Triple* triples, int32_t* tmp_col, double* tmp_val) {
    const int lane = threadIdx.x & 31;
    constexpr int OWN = ROW_SHORT / 32;
    int64_t key[OWN];
    int rank[OWN];
#pragma unroll
    for (int k = 0; k < OWN; k++) {
        key[k] = lane + 32 * k < len ? triples[s + lane + 32 * k].key : INT64_MAX;
        rank[k] = 0;
    }
    for (int j = 0; j < len; j++) {
        const int64_t other = triples[s + j].key;
#pragma unroll
        for (int k = 0; k < OWN; k++) rank[k] += other < key[k];
    }
#pragma unroll
    for (int k = 0; k < OWN; k++)
        if (lane + 32 * k < len) {
            tmp_col[s + rank[k]] = (int32_t)(key[k] >> 32);
            tmp_val[s + rank[k]] = triples[s + lane + 32 * k].w;
        }
    __syncwarp();
    int runs = 0;
    for (int e0 = 0; e0 < len; e0 += 32) {
        const int e = e0 + lane;
        const int32_t c = e < len ? tmp_col[s + e] : 0;
        const bool head = e < len && (e == 0 || tmp_col[s + e - 1] != c);
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        if (head) {
            int h = e + 1;
            while (h < len && tmp_col[s + h] == c) h++;
            triples[s + runs + __popc(heads & ((1u << lane) - 1u))] =
                Triple{c, run_sum([&](int64_t k) { return tmp_val[k]; }, s + e, s + h)};
        }
        runs += __popc(heads);
    }
    __syncwarp();
    for (int k = lane; k < runs; k += 32) {
        tmp_col[s + k] = (int32_t)triples[s + k].key;
        tmp_val[s + k] = triples[s + k].w;
    }
    return runs;
}

// The listed blocks (.x; .y counts their finished turns), a row per block and
// turn, its short rows together in one, a warp each: ranked with the keys staged
// in shared-memory tiles, up to 8 triples per thread and pass, and merged by a
// thread per run; the block that finishes a listed block's last turn moves its
// rows together.  (63 pairs of 64^2 and one of
// 512^2 -> 8^2 in a batch, whose 64 rows of 36,000 triples lie in two blocks of
// 32: 14 ms; with a block for all rows of a listed one 270.  512^2 -> 8^2
// alone 11 and 21 ms.)
constexpr int ROW_TILE = 2048;
__global__ void __launch_bounds__(ORDER_THREADS)
    order_rows_long(const int64_t* __restrict__ row_start, int64_t nrows, int per, int2* __restrict__ long_list,
                    const unsigned* __restrict__ long_count, Triple* triples, int32_t* tmp_col, double* tmp_val,
                    int64_t* row_nnz) {
    __shared__ int64_t tile[ROW_TILE];
    __shared__ int pre[ORDER_ROWS + 1], warp_heads[ORDER_THREADS / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // (rows first: turns of few rows, at the end, leave no SM with more of the long ones)
    const int64_t rows = (int64_t)*long_count * per, items = rows + *long_count;
    for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const bool together = item >= rows;
        int2* listed = long_list + (together ? item - rows : item / per);
        const int64_t r0 = (int64_t)listed->x * per, s0 = row_start[r0];
        const int64_t r1 = r0 + per < nrows ? r0 + per : nrows;
        const int64_t r = together ? r0 : r0 + item % per;
        // the listed block's turns: its long rows, and the short ones together
        const bool mine = r0 + lane < r1 && row_start[r0 + lane + 1] - row_start[r0 + lane] > ROW_SHORT;
        const unsigned longer = __ballot_sync(0xffffffffu, mine);
        if (!together && (r >= r1 || !(longer >> (r - r0) & 1u))) continue;
        if (together)
            for (int q = warp; r0 + q < r1; q += ORDER_THREADS / 32)
                if (!(longer >> q & 1u))
                    row_nnz[r0 + q] = order_short_row(
                        row_start[r0 + q], (int)(row_start[r0 + q + 1] - row_start[r0 + q]), triples, tmp_col, tmp_val);
        const int64_t s = together ? 0 : row_start[r], t = together ? 0 : row_start[r + 1], len = t - s;
        for (int64_t e0 = s; e0 < t; e0 += (int64_t)blockDim.x * 8) {
            int64_t mykey[8];
            int64_t rank[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int64_t e = e0 + threadIdx.x + (int64_t)k * blockDim.x;
                mykey[k] = e < t ? triples[e].key : INT64_MAX;
                rank[k] = 0;
            }
            for (int64_t q0 = 0; q0 < len; q0 += ROW_TILE) {
                const int64_t m = len - q0 < ROW_TILE ? len - q0 : ROW_TILE;
                __syncthreads();
                for (int64_t q = threadIdx.x; q < m; q += blockDim.x) tile[q] = triples[s + q0 + q].key;
                __syncthreads();
                // (eight keys for each read of the tile, or the one of a short row)
                if (t - e0 > blockDim.x) {
                    for (int64_t q = 0; q < m; q++) {
                        const int64_t kq = tile[q];
#pragma unroll
                        for (int k = 0; k < 8; k++) rank[k] += kq < mykey[k];
                    }
                } else {
                    int below = 0;
#pragma unroll 4
                    for (int q = 0; q < (int)m; q++) below += tile[q] < mykey[0];
                    rank[0] += below;
                }
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int64_t e = e0 + threadIdx.x + (int64_t)k * blockDim.x;
                if (e < t) {
                    tmp_col[s + rank[k]] = (int32_t)(mykey[k] >> 32);
                    tmp_val[s + rank[k]] = triples[e].w;
                }
            }
        }
        // a thread adds up each run; the merged row goes through its triples' place
        int runs = 0;
        for (int64_t e0 = s; e0 < t; e0 += blockDim.x) {
            __syncthreads();
            const int64_t e = e0 + threadIdx.x;
            const int32_t c = e < t ? tmp_col[e] : 0;
            const bool head = e < t && (e == s || tmp_col[e - 1] != c);
            const unsigned heads = __ballot_sync(0xffffffffu, head);
            if ((threadIdx.x & 31) == 0) warp_heads[threadIdx.x >> 5] = __popc(heads);
            __syncthreads();
            int at = runs + __popc(heads & ((1u << (threadIdx.x & 31)) - 1u));
            for (int w = 0; w < ORDER_THREADS / 32; w++) {
                at += w < (threadIdx.x >> 5) ? warp_heads[w] : 0;
                runs += warp_heads[w];
            }
            if (head) {
                int64_t h = e + 1;
                while (h < t && tmp_col[h] == c) h++;
                triples[s + at] = Triple{c, run_sum([&](int64_t k) { return tmp_val[k]; }, e, h)};
            }
        }
        __syncthreads();
        for (int k = threadIdx.x; k < runs; k += blockDim.x) {
            tmp_col[s + k] = (int32_t)triples[s + k].key;
            tmp_val[s + k] = triples[s + k].w;
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            if (!together) row_nnz[r] = runs;
            __threadfence();
            last = atomicAdd(&listed->y, 1) == __popc(longer);
            __threadfence();
        }
        __syncthreads();
        if (!last) continue;
        if (threadIdx.x < 32) {
            const int64_t row = r0 + threadIdx.x;
            order_counts(row < r1 ? (int)__ldcg(row_nnz + row) : 0, pre);
        }
        __syncthreads();
        // (entries move towards the front: a pass reads before any of it writes)
        for (int q = 0; r0 + q < r1; q++) {
            const int64_t src = row_start[r0 + q] - pre[q];
            for (int e0 = pre[q]; e0 < pre[q + 1]; e0 += blockDim.x) {
                const int e = e0 + threadIdx.x;
                const bool have = e < pre[q + 1];
                const int32_t c = have ? __ldcg(tmp_col + src + e) : 0;
                const double v = have ? __ldcg(tmp_val + src + e) : 0.0;
                __syncthreads();
                if (have) {
                    tmp_col[s0 + e] = c;
                    tmp_val[s0 + e] = v;
                }
                __syncthreads();
            }
        }
        __syncthreads();
    }
}

// The blocks' merged entries to their place in the CSR.
constexpr int COPY_THREADS = 128;
__global__ void __launch_bounds__(COPY_THREADS)
    copy_blocks(const int64_t* __restrict__ row_start, const int64_t* __restrict__ row_ptr, int64_t nrows, int per,
                const int32_t* __restrict__ tmp_col, const double* __restrict__ tmp_val, int32_t* __restrict__ col,
                double* __restrict__ val) {
    const int64_t r0 = (int64_t)blockIdx.x * per, r1 = r0 + per < nrows ? r0 + per : nrows;
    const int64_t s = row_start[r0], d = row_ptr[r0], n = row_ptr[r1] - d;
    for (int64_t e = threadIdx.x; e < n; e += COPY_THREADS) {
        col[d + e] = tmp_col[s + e];
        val[d + e] = tmp_val[s + e];
    }
}

// One thread per output cell: merge equal input indices of the cell's sorted
// raw entries with the add.reduceat association, first + pairwise(rest),
// writing (col, value) compactly from the bucket start; count them.
// The sorted raw entries arrive as contiguous (input index, value) arrays
// (the bucket sort gathers them while ranking), so each thread reads its
// row's entries in order instead of chasing a permutation.
struct SortedVal {
    const double* val;
    __device__ __forceinline__ double operator()(int64_t k) const { return val[k]; }
};

__global__ void merge_rows(const int64_t* __restrict__ bptr, const int32_t* __restrict__ s_in,
                           const double* __restrict__ s_val, int64_t n_out, int32_t* __restrict__ tmp_col,
                           double* __restrict__ tmp_val, int64_t* __restrict__ row_nnz) {
    SortedVal at{s_val};
    for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < n_out;
         o += (int64_t)gridDim.x * blockDim.x)
        row_nnz[o] = merge_sorted(
                         bptr[o], bptr[o + 1], [&](int64_t k) { return s_in[k]; }, at,
                         [&](int64_t k, int32_t c, double v) {
                             tmp_col[k] = c;
                             tmp_val[k] = v;
                         }) -
                     bptr[o];
}

__global__ void compact_rows(const int64_t* __restrict__ bptr, const int64_t* __restrict__ row_ptr,
                             const int32_t* __restrict__ tmp_col, const double* __restrict__ tmp_val,
                             int64_t n_out, int32_t* __restrict__ col, double* __restrict__ val) {
    for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < n_out;
         o += (int64_t)gridDim.x * blockDim.x) {
        int64_t s = bptr[o], d = row_ptr[o], n = row_ptr[o + 1] - d;
        for (int64_t k = 0; k < n; k++) {
            col[d + k] = tmp_col[s + k];
            val[d + k] = tmp_val[s + k];
        }
    }
}

// Bins of a static grid with bounding box bb: square, sized so that a bin
// holds about one edge along the boundary; at most 1024 a side.
Bins static_bins(const double* bb, int64_t nedges) {
    const double ex = bb[2] - bb[0], ey = bb[3] - bb[1];
    const double ext = ex > ey ? ex : ey;
    int64_t side = nedges / 8;
    if (side < 8) side = 8;
    if (side > 1024) side = 1024;
    const double hbin = ext > 0 && std::isfinite(ext) ? ext / (double)side : 1.0;
    Bins b;
    b.ox = bb[0];
    b.oy = bb[1];
    b.inv_h = 1.0 / hbin;
    b.nbx = (int)std::min<double>(1024.0, std::max(1.0, std::ceil(ex / hbin)));
    b.nby = (int)std::min<double>(1024.0, std::max(1.0, std::ceil(ey / hbin)));
    if (!std::isfinite(ex) || !std::isfinite(ey)) {
        b.nbx = 1;
        b.nby = 1;
    }
    b.ptr = nullptr;
    b.items = nullptr;
    return b;
}

// Batch-wide arrays of the static grids' preparation (PrepGrid)
struct StaticBatch {
    PrepGrid* grids = nullptr;  // [2G]
    Edge* edges = nullptr;
    unsigned* counts = nullptr;
    int64_t* ptr64 = nullptr;
    int32_t* ptr32 = nullptr;
    int32_t* items = nullptr;
    double* bbox_part = nullptr;
    void free(cudaStream_t s) {
        dfree(grids, s);
        dfree(edges, s);
        dfree(counts, s);
        dfree(ptr64, s);
        dfree(ptr32, s);
        dfree(items, s);
        dfree(bbox_part, s);
        *this = StaticBatch();
    }
};

}  // namespace

int cell_area_2d(const double* x, const double* y, int64_t nx, int64_t ny, double* area,
                 cudaStream_t s) {
    int64_t n = (nx - 1) * (ny - 1);
    if (n <= 0) return RG_OK;
    cell_area_kernel<<<grid_for(n, 256), 256, 0, s>>>(x, y, nx, ny, area);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

// Seat lookup for points (the locator entry point): method 0 brute, 1 secant
__global__ void locate_points_kernel(Grid g, const double* px, const double* py, int64_t n,
                                     int method, int64_t* oi, int64_t* oj) {
    int lane = threadIdx.x & 31;
    int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (k >= n) return;
    double x = px[k], y = py[k];
    int64_t i = MAXSIZE, j = MAXSIZE;
    const bool ok = method == 1 && locate_secant_warp(g, x, y, &i, &j);
    if (!ok) locate_brute_warp(g, x, y, &i, &j);
    if (lane == 0) {
        oi[k] = i;
        oj[k] = j;
    }
}

int locate_2d_exact(const double* x, const double* y, int64_t nx, int64_t ny, const double* px,
                    const double* py, int64_t n, int method, int64_t* oi, int64_t* oj,
                    cudaStream_t s) {
    if (n <= 0) return RG_OK;
    locate_points_kernel<<<grid_for(n * 32, 128), 128, 0, s>>>(Grid{x, y, nx, ny}, px, py, n, method,
                                                               oi, oj);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

std::atomic<int64_t> g_sweep_chunk{32};
// two chunks for each thread of the walk (8 blocks of 64 per SM): lengths
// differ, and a second round evens them out (one chunk per thread against two:
// 1024^2 -> 200^2 1.73 and 1.32 ms with the apply, 700^2 -> 500^2 0.93 and 0.89;
// 333x257 and 16 pairs of 32 to 256 the same; 2048^2 is above either)
constexpr int64_t kTargetChunks = 152 * 1024;
constexpr int64_t kMinChunk = 1;

namespace {

// The walk failures a grid's error word records, as a status (message set).
int walk_status(unsigned fl) {
    if (fl & (FLAG_WALK_CAP | FLAG_SEAT_OUTSIDE)) {
        set_error("conservative sweep: %s",
                  (fl & FLAG_WALK_CAP) ? "a grid line exceeded its step cap (degenerate grids?)"
                                       : "a grid line starting inside the grid boundary could "
                                         "not be located in any cell");
        return RG_ERR_WALK;
    }
    return RG_OK;
}

template <typename T>
int upload(T** d, const std::vector<T>& h, cudaStream_t s) {
    RG_TRY(dalloc(d, h.size(), s));
    RG_TRY(small_to_device(*d, h.data(), sizeof(T) * h.size(), s));
    return RG_OK;
}

// Small arrays that go to the device together: one allocation, one copy.
struct Pack {
    std::vector<unsigned char> bytes;
    unsigned char* dev = nullptr;
    size_t add(const void* src, size_t n) {  // null: zeros
        const size_t at = (bytes.size() + 15) & ~(size_t)15;
        bytes.resize(at + n, 0);
        if (src) memcpy(bytes.data() + at, src, n);
        return at;
    }
    template <typename T>
    size_t add(const std::vector<T>& v) {
        return add(v.data(), sizeof(T) * v.size());
    }
    int to_device(cudaStream_t s) {
        RG_TRY(dalloc(&dev, bytes.size(), s));
        return small_to_device(dev, bytes.data(), bytes.size(), s);
    }
    template <typename T>
    T* at(size_t offset) const {
        return reinterpret_cast<T*>(dev + offset);
    }
};

// A count on the device and the grids' error words, which follow it, by one copy.
int count_and_flags(const int64_t* total_dev, int64_t* total, std::vector<unsigned>& fl, cudaStream_t s) {
    std::vector<unsigned char> buf(sizeof(int64_t) + sizeof(unsigned) * fl.size());
    RG_TRY(small_to_host(buf.data(), total_dev, buf.size(), s));
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_error("conservative sweep: %s", cudaGetErrorString(e));
        return RG_ERR_CUDA;
    }
    memcpy(total, buf.data(), sizeof(int64_t));
    memcpy(fl.data(), buf.data() + sizeof(int64_t), sizeof(unsigned) * fl.size());
    return RG_OK;
}

// One thread per line over all lines of the batch, count then write
// (synchronises once; total_dev with the error words behind it).  fl receives every grid's error word.
int sweep_lines(const Batch& B, int64_t lines, const Seat* seats, int64_t* total_dev, cudaStream_t s,
                int32_t** raw_in, int32_t** raw_out, double** raw_val, int64_t* nraw_out, std::vector<unsigned>& fl) {
    int64_t *counts = nullptr, *offsets = nullptr;
    int st = RG_OK;
    do {
        if ((st = dalloc(&counts, (size_t)lines + 1, s))) break;
        if ((st = dalloc(&offsets, (size_t)lines + 1, s))) break;
        walk_kernel<false><<<grid_for(lines, 64), 64, 0, s>>>(B, seats, counts, nullptr, nullptr, nullptr, nullptr);
        zero_async(counts + lines, sizeof(int64_t), s);
        if ((st = exclusive_scan_i64(counts, offsets, lines + 1, total_dev, s))) break;
        int64_t nraw = 0;
        if ((st = count_and_flags(total_dev, &nraw, fl, s))) break;
        if (nraw >= (int64_t)UINT32_MAX) {
            set_error("conservative sweep: %lld raw entries exceed 2^32", (long long)nraw);
            st = RG_ERR_UNSUPPORTED;
            break;
        }
        if ((st = dalloc(raw_in, (size_t)nraw, s))) break;
        if ((st = dalloc(raw_out, (size_t)nraw, s))) break;
        if ((st = dalloc(raw_val, (size_t)nraw, s))) break;
        walk_kernel<true><<<grid_for(lines, 64), 64, 0, s>>>(B, seats, nullptr, offsets, *raw_in, *raw_out, *raw_val);
        *nraw_out = nraw;
    } while (0);
    dfree(counts, s);
    dfree(offsets, s);
    return st;
}

// The triples merged by output row straight from the chunks' slots
// (slot_count_rows, slot_scatter_rows, order_rows): row_start[n_rows + 1] of
// the buckets, the rows' merged counts, and the merged entries of every
// `per` rows from their first bucket's start on.
struct MergedRows {
    int64_t n_rows = 0;
    int per = 0;
    int64_t* row_start = nullptr;
    int64_t* row_nnz = nullptr;
    int32_t* col = nullptr;
    double* val = nullptr;
};

// Chunked walk over all lines of the batch (see chunk_walk_kernel), its
// triples left merged by output row in *rows.  Sets *nraw_out to -1 (and
// frees everything) when a chunk needed more slots than it was given or the
// slots would not fit; fl receives every grid's error word.

int sweep_chunked(Batch& B, const std::vector<SweepParams>& P, const std::vector<double>& bbox_h,
                  Seat* seats, int64_t lines, int64_t* total_dev, cudaStream_t s, int64_t* nraw_out,
                  std::vector<unsigned>& fl, unsigned char** plans_dev, MergedRows* rows) {
    const int G = B.G;
    // sweep segments per chunk: rg_set_sweep_chunk (default 32), the
    // RG_SWEEP_CHUNK environment variable overriding it (0 walks whole lines)
    int64_t ch = g_sweep_chunk.load();
    if (const char* env = getenv("RG_SWEEP_CHUNK")) {
        ch = atoll(env);
    } else if (ch > kMinChunk) {
        // Small batches: shorter chunks, so that the walk still has about
        // kTargetChunks chunks (each is one thread's sequential walk; a 128^2
        // pair in chunks of 32 segments keeps 2,000 threads busy for 0.7 ms), down to one segment (a start costs little beside the
        // walk of a segment; 64^2 -> 48^2: walk 100 -> 34 us).  Every chunk length gives the same
        // triples in the same order.
        int64_t segments = 0;
        for (int g = 0; g < G; g++)
            for (int f = 0; f < 4; f++) segments += P[g].fam[f].lines * (P[g].fam[f].len - 1);
        const int64_t fit = (segments + kTargetChunks - 1) / kTargetChunks;
        ch = std::min<int64_t>(ch, std::max<int64_t>(kMinChunk, fit));
    }
    *nraw_out = -1;
    if (ch <= 0) return RG_OK;
    // fault injection for tests: RG_FAULT_CHUNK_SLOTS caps the piece slots
    // a chunk gets, so chunks overflow and the build takes its recovery path
    // (whole-line walks, which count exactly); the weights do not change
    int64_t slot_cap = INT64_MAX;
    if (const char* env = getenv("RG_FAULT_CHUNK_SLOTS")) slot_cap = std::max<int64_t>(1, atoll(env));
    // Slots per chunk: those of twice its segments (4 to 32) at the crossings of
    // grids of even cells, and 48, since a short chunk has nothing to set off a
    // segment of graded grids against that crosses many cells, and one chunk that
    // overflows sends the build to whole lines.  (Output lines at s |x|^2 from 512^2
    // vertices: 1.8 ms with chunks of four segments and more, 7.4 with the slots of
    // shorter ones alone, 1.2 so; 1024^2: 3.3, 15.3 and 1.9.)
    const int64_t span = ch < 32 ? std::min<int64_t>(32, std::max<int64_t>(4, 2 * ch)) : ch, slack = ch < 32 ? 48 : 16;
    std::vector<ChunkPlan> C((size_t)G);
    std::vector<int64_t> chunk_base((size_t)G + 1, 0);
    int64_t chunks = 0, slots = 0;
    for (int g = 0; g < G; g++) {
        ChunkPlan& c = C[g];
        memset(&c, 0, sizeof(c));
        c.ch = ch;
        chunk_base[g] = chunks;
        const double* bb = bbox_h.data() + 8 * g;
        for (int f = 0; f < 4; f++) {
            const Family& F = P[g].fam[f];
            const Static& S = P[g].st[F.st];
            const double* bs = F.sweep_input ? bb : bb + 4;  // sweep grid's box
            const double* bt = F.sweep_input ? bb + 4 : bb;  // static grid's box
            double seg = fmax(bs[2] - bs[0], bs[3] - bs[1]) / (double)(F.len - 1 > 0 ? F.len - 1 : 1);
            double dens = fmax((double)S.ncx / fmax(bt[2] - bt[0], 1e-300), (double)S.ncy / fmax(bt[3] - bt[1], 1e-300));
            double cross = 2.0 * ceil(1.5 * seg * dens) + 2.0;
            if (!(cross < 1e6)) cross = 1e6;
            c.nc[f] = (F.len - 1 + ch - 1) / ch;
            c.chunk_base[f] = chunks;
            c.cap[f] = std::min<int64_t>(span * (1 + (int64_t)cross) + slack, slot_cap);
            c.slot_base[f] = slots;
            chunks += F.lines * c.nc[f];
            slots += F.lines * c.nc[f] * c.cap[f];
        }
        c.chunk_base[4] = chunks;
    }
    chunk_base[G] = chunks;
    // too big: walk lines (a slot: a piece and its two triples' places)
    constexpr int64_t SLOT_BYTES = 2 * sizeof(int32_t) + sizeof(double) + sizeof(uint2);
    if (slots > ((int64_t)24 << 30) / SLOT_BYTES) return RG_OK;

    WalkState *starts = nullptr, *ends = nullptr;
    int64_t *counts = nullptr, *offsets = nullptr;
    int32_t *s_in = nullptr, *s_out = nullptr;
    double* s_val = nullptr;
    uint2* s_pos = nullptr;
    unsigned long long* n_rep = nullptr;
    int st = RG_OK;
    bool overflow = false;
    do {
        // the plans, and two counts: chunks repaired, next chunk of the walk
        Pack pack;
        const size_t plans_at = pack.add(C), base_at = pack.add(chunk_base);
        const size_t rep_at = pack.add(nullptr, 2 * sizeof(unsigned long long));
        st = pack.to_device(s);
        *plans_dev = pack.dev;
        if (st) break;
        B.C = pack.at<ChunkPlan>(plans_at);
        B.chunk_base = pack.at<int64_t>(base_at);
        n_rep = pack.at<unsigned long long>(rep_at);
        if ((st = dalloc(&starts, (size_t)chunks, s))) break;
        if ((st = dalloc(&ends, (size_t)chunks, s))) break;
        if ((st = dalloc(&counts, (size_t)chunks + 1, s))) break;
        if ((st = dalloc(&offsets, (size_t)chunks + 1, s))) break;
        if ((st = dalloc(&s_in, (size_t)slots, s))) break;
        if ((st = dalloc(&s_out, (size_t)slots, s))) break;
        if ((st = dalloc(&s_val, (size_t)slots, s))) break;
        if ((st = dalloc(&s_pos, (size_t)slots, s))) break;
        const unsigned seat_blocks = grid_for(lines * 32, 128);
        chunk_seat_kernel<<<seat_blocks + grid_for(chunks + 1, 128), 128, 0, s>>>(B, seat_blocks, seats, starts, counts);
        {
            // resident blocks only: 8 blocks of 64 threads per SM
            const unsigned blocks = std::min<unsigned>(grid_for(chunks, 64), 152u * 8u);
            chunk_walk_kernel<<<blocks, 64, 0, s>>>(B, starts, ends, counts, s_in, s_out, s_val, n_rep + 1);
        }
        chunk_repair_kernel<<<grid_for(lines * 32, 128), 128, 0, s>>>(B, starts, ends, counts, s_in, s_out, s_val, n_rep);
        if ((st = exclusive_scan_i64(counts, offsets, chunks + 1, total_dev, s))) break;
        int64_t nraw = 0;  // pieces; up to two triples each
        if ((st = count_and_flags(total_dev, &nraw, fl, s))) break;
        nraw *= 2;
        bool cap = false;
        for (unsigned f : fl) cap = cap || (f & FLAG_CAPACITY);
        if (cap) {
            overflow = true;
            zero_async(B.flags, sizeof(unsigned) * fl.size(), s);
            break;
        }
        if (nraw >= (int64_t)UINT32_MAX) {  // raw positions past 32 bits: the whole-line walk counts the triples
            overflow = true;
            break;
        }
        {
            // order the triples by output row from the slots
            const int64_t nr = rows->n_rows;
            unsigned *rowc = nullptr, *long_count = nullptr;  // (one allocation)
            Triple* triples = nullptr;
            int2* long_list = nullptr;
            do {
                if ((st = dalloc(&rows->row_start, (size_t)nr + 1, s))) break;
                if ((st = dalloc(&rows->row_nnz, (size_t)nr + 1, s))) break;
                if ((st = dalloc(&rows->col, (size_t)nraw, s))) break;
                if ((st = dalloc(&rows->val, (size_t)nraw, s))) break;
                if ((st = dalloc(&rowc, (size_t)nr + 2, s))) break;
                long_count = rowc + nr + 1;
                rows->per = order_rows_per_block(nraw, nr);
                if ((st = dalloc(&long_list, (size_t)(nr / rows->per + 1), s))) break;
                if ((st = dalloc(&triples, (size_t)nraw, s))) break;
                zero_async(rowc, sizeof(unsigned) * (nr + 2), s);
                // lanes per chunk for the pieces it holds on average (the lines at
                // 20 and 10 against 48 and 24, builds with their applies: 512^2 ->
                // 384^2 688 and 677 us, 700^2 -> 500^2 911 and 893, 1024^2 -> 768^2
                // 1.50 and 1.47 ms, 2048^2 -> 1536^2 the same)
                const int64_t mean = nraw / (2 * chunks);
                const int lanes = mean > 48 ? 32 : mean > 24 ? 16 : 8;
                const unsigned gc = grid_for(chunks * lanes, 256);
                const auto count = lanes == 32 ? slot_count_rows<32> : lanes == 16 ? slot_count_rows<16> : slot_count_rows<8>;
                const auto scatter = lanes == 32   ? slot_scatter_rows<32>
                                     : lanes == 16 ? slot_scatter_rows<16>
                                                   : slot_scatter_rows<8>;
                count<<<gc, 256, 0, s>>>(B, counts, s_in, s_out, rowc, s_pos);
                if ((st = exclusive_scan_u32_to_i64(rowc, rows->row_start, nr + 1, nullptr, s))) break;
                scatter<<<gc, 256, 0, s>>>(B, counts, offsets, s_in, s_out, s_val, s_pos, rows->row_start, triples);
                const unsigned blocks = grid_for(nr, rows->per);
                const auto order = rows->per == 32 ? order_rows<32> : rows->per == 8 ? order_rows<8> : order_rows<2>;
                order<<<blocks, ORDER_THREADS, 0, s>>>(rows->row_start, nr, triples, rows->col, rows->val,
                                                       rows->row_nnz, long_list, long_count);
                order_rows_long<<<std::min(grid_for(2 * nr, 1), 152u * 8u), ORDER_THREADS, 0, s>>>(rows->row_start, nr, rows->per, long_list,
                                                                            long_count, triples, rows->col, rows->val,
                                                                            rows->row_nnz);
            } while (0);
            dfree(rowc, s);
            dfree(long_list, s);
            dfree(triples, s);
            if (st) break;
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_error("conservative sweep (compaction): %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }
        *nraw_out = nraw;
    } while (0);
    dfree(starts, s);
    dfree(ends, s);
    dfree(counts, s);
    dfree(offsets, s);
    dfree(s_in, s);
    dfree(s_out, s);
    dfree(s_val, s);
    dfree(s_pos, s);
    if (overflow) *nraw_out = -1;
    return st;
}

// Per-grid sizes of the merged CSR: nnz_base[g] = row_ptr[out_base[g]].
__global__ void nnz_bases(const int64_t* __restrict__ row_ptr, const int64_t* __restrict__ out_base,
                          const unsigned* __restrict__ flags, int G, int64_t* __restrict__ nnz_base) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= G; g += gridDim.x * blockDim.x) {
        nnz_base[g] = row_ptr[out_base[g]];
        if (g < G) nnz_base[G + 1 + g] = flags[g];  // the grids' error words behind them
    }
}

// Copy every grid's rows and entries of the merged CSR to its own arrays.
__global__ void split_rows(const int64_t* __restrict__ row_ptr, const int64_t* __restrict__ out_base,
                           const int64_t* __restrict__ nnz_base, int G, int64_t* const* __restrict__ dst_row_ptr) {
    const int64_t n = out_base[G];
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        const int g = pair_of(out_base, G, r);
        const int64_t local = r - out_base[g];
        dst_row_ptr[g][local] = row_ptr[r] - nnz_base[g];
        if (r + 1 == out_base[g + 1]) dst_row_ptr[g][local + 1] = row_ptr[r + 1] - nnz_base[g];
    }
}
__global__ void split_entries(const int32_t* __restrict__ col, const double* __restrict__ val,
                              const int64_t* __restrict__ nnz_base, int G, int32_t* const* __restrict__ dst_col,
                              double* const* __restrict__ dst_val) {
    const int64_t n = nnz_base[G];
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int g = pair_of(nnz_base, G, k);
        const int64_t local = k - nnz_base[g];
        dst_col[g][local] = col[k];
        dst_val[g][local] = val[k];
    }
}

}  // namespace

// Conservative weights of G grid pairs in one pass: every stage runs once
// over all pairs (their lines, chunks and output rows concatenated), and the
// batch synchronises with the host five times whatever G is.  W[g] receives
// pair g's CSR when status[g] is RG_OK; a pair whose sweep fails (degenerate
// grids) gets its error in status[g] and leaves the others unaffected.
int build_batch(const PairSpec* pairs, int G, cudaStream_t s, rg_weights_s** W, int* status) {
    RG_CHECK(G >= 1, RG_ERR_ARG, "conservative batch: no grid pairs");
    std::vector<int64_t> in_base((size_t)G + 1, 0), out_base((size_t)G + 1, 0), line_base((size_t)G + 1, 0);
    for (int g = 0; g < G; g++) {
        const PairSpec& q = pairs[g];
        RG_CHECK(q.nxi >= 2 && q.nyi >= 2 && q.nxo >= 2 && q.nyo >= 2, RG_ERR_ARG,
                 "conservative 2D grids need at least 2 vertices per axis");
        const int64_t n_in = (q.nxi - 1) * (q.nyi - 1), n_out = (q.nxo - 1) * (q.nyo - 1);
        in_base[g + 1] = in_base[g] + n_in;
        out_base[g + 1] = out_base[g] + n_out;
        // lines of the four families: output rows/columns, then input rows/columns
        line_base[g + 1] = line_base[g] + q.nyo + q.nxo + q.nyi + q.nxi;
        status[g] = RG_OK;
    }
    RG_CHECK(in_base[G] < INT32_MAX && out_base[G] < INT32_MAX, RG_ERR_UNSUPPORTED,
             "grids above 2^31 cells (in a batch, in total) are not supported");
    const int64_t lines = line_base[G], n_out_all = out_base[G];

    int st = RG_OK;
    double2* area_in = nullptr;
    double* bbox_d = nullptr;
    StaticBatch SB;
    int64_t* totals = nullptr;
    unsigned char* head_dev = nullptr;  // the sweep parameters, bases, total and error words
    const int64_t* out_base_dev = nullptr;
    unsigned char* plans_dev = nullptr;
    Seat* seats = nullptr;
    int64_t* total_dev = nullptr;
    unsigned* flags = nullptr;
    int32_t *raw_in = nullptr, *raw_out = nullptr, *sorted_in = nullptr;
    double* sorted_val = nullptr;
    double* raw_val = nullptr;
    int64_t* skey = nullptr;
    int64_t* bucket_ptr = nullptr;
    uint32_t* perm = nullptr;
    int32_t* tmp_col = nullptr;
    double* tmp_val = nullptr;
    int64_t* row_nnz = nullptr;
    int64_t* row_ptr = nullptr;
    int32_t* col = nullptr;
    double* val = nullptr;
    int64_t* nnz_base_dev = nullptr;
    void** dst_dev = nullptr;  // [3G]: row_ptr, col, val pointers of every grid

    do {
        // static grids: the input and the output grid of every pair.  Areas
        // of the input cells, bounding boxes and boundary edges of all grids
        // (sync 1 reads the boxes)
        const int NG = 2 * G;
        std::vector<PrepGrid> PG((size_t)NG);
        int64_t nedges_all = 0, max_verts = 0;
        for (int k = 0; k < NG; k++) {
            const PairSpec& q = pairs[k >> 1];
            PrepGrid& r = PG[k];
            memset(&r, 0, sizeof(PrepGrid));
            r.g = (k & 1) ? Grid{q.xo, q.yo, q.nxo, q.nyo} : Grid{q.xi, q.yi, q.nxi, q.nyi};
            r.cell_base = (k & 1) ? 0 : in_base[k >> 1];
            r.edge_base = nedges_all;
            nedges_all += 2 * (r.g.nx - 1) + 2 * (r.g.ny - 1);
            max_verts = std::max(max_verts, r.g.nx * r.g.ny);
        }
        // blocks per grid for the boxes: about 4 vertices a thread, 1..512
        const int nparts = (int)std::min<int64_t>(512, std::max<int64_t>(1, (max_verts + 1023) / 1024));
        if ((st = upload(&SB.grids, PG, s))) break;
        if ((st = dalloc(&area_in, (size_t)in_base[G], s))) break;
        if ((st = dalloc(&bbox_d, (size_t)4 * NG, s))) break;
        if ((st = dalloc(&SB.bbox_part, (size_t)4 * NG * nparts, s))) break;
        if ((st = dalloc(&SB.edges, (size_t)nedges_all, s))) break;
        const unsigned box_blocks = (unsigned)(NG * nparts), edge_blocks = grid_for(nedges_all, 256);
        prepare_batch<<<box_blocks + edge_blocks + grid_for(in_base[G], 256), 256, 0, s>>>(
            SB.grids, G, box_blocks, nparts, SB.bbox_part, edge_blocks, nedges_all, SB.edges, in_base[G], area_in);
        bbox_combine_batch<<<grid_for((int64_t)NG * 32, 128), 128, 0, s>>>(SB.bbox_part, nparts, NG, bbox_d);
        std::vector<double> bbox_h((size_t)4 * NG);
        small_to_host(bbox_h.data(), bbox_d, sizeof(double) * 4 * NG, s);
        cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error("conservative build: %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }

        // bins of every static grid: count the edges of each bin, one scan
        // over the slots of all grids (sync 2 reads the item total), file
        int64_t nslots = 0;
        for (int k = 0; k < NG; k++) {
            PrepGrid& r = PG[k];
            r.b = static_bins(bbox_h.data() + 4 * k, 2 * (r.g.nx - 1) + 2 * (r.g.ny - 1));
            r.bin_base = nslots;
            nslots += (int64_t)r.b.nbx * r.b.nby + 1;
        }
        if ((st = small_to_device(SB.grids, PG.data(), sizeof(PrepGrid) * PG.size(), s))) break;
        if ((st = dalloc(&totals, 1, s))) break;
        if ((st = dalloc(&SB.counts, (size_t)nslots, s))) break;
        if ((st = dalloc(&SB.ptr64, (size_t)nslots, s))) break;
        if ((st = dalloc(&SB.ptr32, (size_t)nslots, s))) break;
        if ((st = zero_async(SB.counts, sizeof(unsigned) * nslots, s))) break;
        bin_edges_batch<false><<<grid_for(nedges_all, 128), 128, 0, s>>>(SB.grids, NG, SB.edges, nedges_all,
                                                                          SB.counts, nullptr, nullptr);
        if ((st = exclusive_scan_u32_to_i64(SB.counts, SB.ptr64, nslots, totals, s))) break;
        int64_t nitems = 0;
        small_to_host(&nitems, totals, sizeof(int64_t), s);
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error("conservative build: %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }
        if (nitems >= (int64_t)INT32_MAX) {
            set_error("conservative build: %lld binned boundary edges exceed 2^31", (long long)nitems);
            st = RG_ERR_UNSUPPORTED;
            break;
        }
        if ((st = dalloc(&SB.items, (size_t)nitems, s))) break;
        if ((st = zero_async(SB.counts, sizeof(unsigned) * nslots, s))) break;
        bin_edges_batch<true><<<grid_for(nedges_all, 128), 128, 0, s>>>(SB.grids, NG, SB.edges, nedges_all,
                                                                         SB.counts, SB.items, SB.ptr64);
        i64_to_i32<<<grid_for(nslots, 256), 256, 0, s>>>(SB.ptr64, SB.ptr32, nslots);
        e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_error("conservative build (static grids): %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }
        std::vector<SweepParams> P((size_t)G);
        for (int g = 0; g < G; g++) {
            memset(&P[g], 0, sizeof(SweepParams));
            for (int side = 0; side < 2; side++) {
                const PrepGrid& r = PG[2 * g + side];
                const double* bb = bbox_h.data() + 4 * (2 * g + side);
                Static& S = P[g].st[side];
                S.g = r.g;
                S.ncx = r.g.nx - 1;
                S.ncy = r.g.ny - 1;
                S.blx = bb[0];
                S.bly = bb[1];
                S.bux = bb[2];
                S.buy = bb[3];
                S.nbound = 2 * S.ncx + 2 * S.ncy;
                S.edges = SB.edges + r.edge_base;
                S.bins = r.b;
                S.bins.ptr = SB.ptr32 + r.bin_base;
                S.bins.items = SB.items;
            }
        }

        // sweep families in upstream order: sweep output (axis 0, 1), sweep
        // input (axis 0, 1); line bases global across the batch
        for (int g = 0; g < G; g++) {
            const PairSpec& q = pairs[g];
            int64_t base = line_base[g];
            for (int k = 0; k < 4; k++) {
                Family& F = P[g].fam[k];
                F.sweep_input = k >= 2;
                F.axis = k & 1;
                F.sweep = F.sweep_input ? Grid{q.xi, q.yi, q.nxi, q.nyi} : Grid{q.xo, q.yo, q.nxo, q.nyo};
                F.st = F.sweep_input ? 1 : 0;
                F.transposed = F.axis == 0;
                F.lines = F.axis == 0 ? F.sweep.ny : F.sweep.nx;
                F.len = F.axis == 0 ? F.sweep.nx : F.sweep.ny;
                F.line_base = base;
                base += F.lines;
            }
            P[g].total_lines = base;
            P[g].area_in = area_in + in_base[g];
            P[g].w_in = q.w_in;
            P[g].ncy_in = q.nyi - 1;
            P[g].ncy_out = q.nyo - 1;
        }
        Pack pack;
        const size_t P_at = pack.add(P), line_at = pack.add(line_base), out_at = pack.add(out_base);
        const size_t total_at = pack.add(nullptr, sizeof(int64_t) + sizeof(unsigned) * G);
        st = pack.to_device(s);
        head_dev = pack.dev;
        if (st) break;
        out_base_dev = pack.at<int64_t>(out_at);
        total_dev = pack.at<int64_t>(total_at);
        flags = pack.at<unsigned>(total_at + sizeof(int64_t));
        Batch B;
        B.P = pack.at<SweepParams>(P_at);
        B.C = nullptr;
        B.line_base = pack.at<int64_t>(line_at);
        B.chunk_base = nullptr;
        B.out_base = out_base_dev;
        B.flags = flags;
        B.G = G;

        // seats and the sweep (sync 3)
        if ((st = dalloc(&seats, (size_t)lines, s))) break;
        std::vector<unsigned> fl((size_t)G, 0u);
        int64_t nraw = 0;
        MergedRows rows;
        rows.n_rows = n_out_all;
        st = sweep_chunked(B, P, bbox_h, seats, lines, total_dev, s, &nraw, fl, &plans_dev, &rows);
        bucket_ptr = rows.row_start;
        row_nnz = rows.row_nnz;
        tmp_col = rows.col;
        tmp_val = rows.val;
        if (st) break;
        const bool merged = bucket_ptr != nullptr;
        if (nraw < 0) {
            // a chunk overflowed its slots, or lines are not cut: walk whole lines
            seat_kernel<<<grid_for(lines * 32, 128), 128, 0, s>>>(B, seats);
            if ((st = sweep_lines(B, lines, seats, total_dev, s, &raw_in, &raw_out, &raw_val, &nraw, fl))) break;
        }
        for (int g = 0; g < G; g++) status[g] = walk_status(fl[g]);

        // merge: the triples in output-row order (sync 4 for the entry count;
        // the per-grid sizes come with it).  The chunked walk orders them from
        // its slots; otherwise one bucket sort over the output rows of the
        // whole batch, which also lays the entries' input indices and values
        // out in sorted order, so the merge reads them contiguously.
        if (bucket_ptr == nullptr) {
            if ((st = dalloc(&skey, (size_t)nraw, s))) break;
            if ((st = dalloc(&bucket_ptr, (size_t)n_out_all + 1, s))) break;
            if ((st = dalloc(&perm, (size_t)nraw, s))) break;
            if (nraw > 0)
                make_keys<<<grid_for(nraw, 256) > 8192 ? 8192 : grid_for(nraw, 256), 256, 0, s>>>(raw_in, nraw,
                                                                                                   skey);
            if ((st = dalloc(&sorted_in, (size_t)nraw, s))) break;
            if ((st = dalloc(&sorted_val, (size_t)nraw, s))) break;
            if ((st = bucket_sort(raw_out, skey, nraw, n_out_all, bucket_ptr, perm, flags, s, raw_val, sorted_in,
                                  sorted_val)))
                break;
            dfree(skey, s);
            skey = nullptr;
            dfree(raw_in, s);
            dfree(raw_out, s);
            dfree(raw_val, s);
            raw_in = raw_out = nullptr;
            raw_val = nullptr;
        }
        if (!merged) {
            if ((st = dalloc(&tmp_col, (size_t)nraw, s))) break;
            if ((st = dalloc(&tmp_val, (size_t)nraw, s))) break;
            if ((st = dalloc(&row_nnz, (size_t)n_out_all + 1, s))) break;
            merge_rows<<<grid_for(n_out_all, 128), 128, 0, s>>>(bucket_ptr, sorted_in, sorted_val, n_out_all, tmp_col,
                                                                tmp_val, row_nnz);
            zero_async(row_nnz + n_out_all, sizeof(int64_t), s);
        }
        if ((st = dalloc(&row_ptr, (size_t)n_out_all + 1, s))) break;
        if ((st = exclusive_scan_i64(row_nnz, row_ptr, n_out_all + 1, total_dev, s))) break;
        if ((st = dalloc(&nnz_base_dev, 2 * (size_t)G + 1, s))) break;
        nnz_bases<<<grid_for(G + 1, 128), 128, 0, s>>>(row_ptr, out_base_dev, flags, G, nnz_base_dev);
        std::vector<int64_t> nnz_base(2 * (size_t)G + 1, 0);  // the bases, then the error words
        small_to_host(nnz_base.data(), nnz_base_dev, sizeof(int64_t) * nnz_base.size(), s);
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error("conservative build (merge): %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }
        for (int g = 0; g < G; g++)
            if (status[g] == RG_OK && (nnz_base[G + 1 + g] & FLAG_CAPACITY)) {
                set_error("conservative sweep: the write walk disagreed with the count walk");
                status[g] = RG_ERR_WALK;
            }
        const int64_t nnz = nnz_base[G];
        if ((st = dalloc(&col, (size_t)nnz, s))) break;
        if ((st = dalloc(&val, (size_t)nnz, s))) break;
        if (merged)
            copy_blocks<<<grid_for(n_out_all, rows.per), COPY_THREADS, 0, s>>>(bucket_ptr, row_ptr, n_out_all, rows.per,
                                                                               tmp_col, tmp_val, col, val);
        else
            compact_rows<<<grid_for(n_out_all, 128), 128, 0, s>>>(bucket_ptr, row_ptr, tmp_col, tmp_val, n_out_all, col,
                                                                  val);
        e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_error("conservative build: %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }

        // hand every grid its CSR: a single pair takes the arrays as they
        // are, several get their own copies (no synchronisation)
        auto fill_handle = [&](int g) {
            const PairSpec& q = pairs[g];
            W[g]->n_in = in_base[g + 1] - in_base[g];
            W[g]->n_out = out_base[g + 1] - out_base[g];
            W[g]->nnz = nnz_base[g + 1] - nnz_base[g];
            W[g]->out_shape0 = q.nxo - 1;
            W[g]->out_shape1 = q.nyo - 1;
            W[g]->in_shape0 = q.nxi - 1;
            W[g]->in_shape1 = q.nyi - 1;
        };
        if (G == 1) {
            W[0]->row_ptr = row_ptr;
            W[0]->col = col;
            W[0]->val = val;
            fill_handle(0);
            row_ptr = nullptr;
            col = nullptr;
            val = nullptr;
            break;
        }
        std::vector<void*> dst((size_t)3 * G, nullptr);
        for (int g = 0; g < G && st == RG_OK; g++) {
            if (status[g] != RG_OK) continue;
            fill_handle(g);
            if ((st = dalloc(&W[g]->row_ptr, (size_t)W[g]->n_out + 1, s))) break;
            if ((st = dalloc(&W[g]->col, (size_t)W[g]->nnz, s))) break;
            if ((st = dalloc(&W[g]->val, (size_t)W[g]->nnz, s))) break;
            dst[g] = W[g]->row_ptr;
            dst[G + g] = W[g]->col;
            dst[2 * G + g] = W[g]->val;
        }
        if (st) break;
        // grids that failed get scratch destinations: their rows are copied and dropped
        int64_t max_rows = 0, max_nnz = 0;
        for (int g = 0; g < G; g++)
            if (dst[g] == nullptr) {
                max_rows = std::max(max_rows, out_base[g + 1] - out_base[g] + 1);
                max_nnz = std::max(max_nnz, nnz_base[g + 1] - nnz_base[g]);
            }
        int64_t* junk_rows = nullptr;
        int32_t* junk_col = nullptr;
        double* junk_val = nullptr;
        if (max_rows > 0) {
            if ((st = dalloc(&junk_rows, (size_t)max_rows, s))) break;
            if ((st = dalloc(&junk_col, (size_t)std::max<int64_t>(max_nnz, 1), s))) break;
            if ((st = dalloc(&junk_val, (size_t)std::max<int64_t>(max_nnz, 1), s))) break;
            for (int g = 0; g < G; g++)
                if (dst[g] == nullptr) {
                    dst[g] = junk_rows;
                    dst[G + g] = junk_col;
                    dst[2 * G + g] = junk_val;
                }
        }
        if ((st = upload(&dst_dev, dst, s))) break;
        split_rows<<<grid_for(n_out_all, 256) > 8192 ? 8192 : grid_for(n_out_all, 256), 256, 0, s>>>(
            row_ptr, out_base_dev, nnz_base_dev, G, (int64_t* const*)dst_dev);
        if (nnz > 0)
            split_entries<<<grid_for(nnz, 256) > 8192 ? 8192 : grid_for(nnz, 256), 256, 0, s>>>(
                col, val, nnz_base_dev, G, (int32_t* const*)(dst_dev + G), (double* const*)(dst_dev + 2 * G));
        dfree(junk_rows, s);
        dfree(junk_col, s);
        dfree(junk_val, s);
        e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_error("conservative build (split): %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }
    } while (0);

#ifdef RG_DEBUG
    if (st == RG_OK) {  // (a build that fails otherwise leaves the word to the next)
        unsigned dbg = 0;
        const unsigned zero = 0;
        cudaMemcpyFromSymbolAsync(&dbg, g_debug_flags, sizeof(unsigned), 0, cudaMemcpyDeviceToHost, s);
        cudaMemcpyToSymbolAsync(g_debug_flags, &zero, sizeof(unsigned), 0, cudaMemcpyHostToDevice, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) {
            set_error("conservative build (debug flags): %s", cudaGetErrorString(cudaGetLastError()));
            st = RG_ERR_CUDA;
        } else if (dbg & FLAG_BOUNDS) {
            set_error("conservative build: debug bounds check: a grid read fell outside its array");
            for (int g = 0; g < G; g++) status[g] = RG_ERR_WALK;
        }
    }
#endif

    dfree(area_in, s);
    dfree(bbox_d, s);
    SB.free(s);
    dfree(totals, s);
    dfree(head_dev, s);
    dfree(plans_dev, s);
    dfree(seats, s);
    dfree(raw_in, s);
    dfree(raw_out, s);
    dfree(raw_val, s);
    dfree(sorted_in, s);
    dfree(sorted_val, s);
    dfree(skey, s);
    dfree(bucket_ptr, s);
    dfree(perm, s);
    dfree(tmp_col, s);
    dfree(tmp_val, s);
    dfree(row_nnz, s);
    dfree(row_ptr, s);
    dfree(col, s);
    dfree(val, s);
    dfree(nnz_base_dev, s);
    dfree(dst_dev, s);
    return st;
}

int build_conservative_2d(const double* xi, const double* yi, int64_t nxi, int64_t nyi,
                          const double* xo, const double* yo, int64_t nxo, int64_t nyo,
                          const double* w_in, cudaStream_t s, rg_weights_s* W) {
    PairSpec q{xi, yi, nxi, nyi, xo, yo, nxo, nyo, w_in};
    int status = RG_OK;
    RG_TRY(build_batch(&q, 1, s, &W, &status));
    return status;
}

}  // namespace rg

extern "C" int rg_set_sweep_chunk(int64_t segments) {
    RG_CHECK(segments >= 0 && segments <= (1 << 20), RG_ERR_ARG, "rg_set_sweep_chunk: %lld out of range",
             (long long)segments);
    rg::g_sweep_chunk.store(segments);
    return RG_OK;
}

#ifdef RG_DEBUG
// Debug builds, for tests of the reporting: sets the bounds word as a read
// outside an array does.
extern "C" int rg_debug_out_of_bounds() {
    const unsigned word = rg::FLAG_BOUNDS;
    RG_CUDA(cudaMemcpyToSymbol(rg::g_debug_flags, &word, sizeof(word)));
    return RG_OK;
}
#endif
