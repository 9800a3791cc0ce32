// Adjoint of the 2D conservative weights with respect to the output-grid
// vertex coordinates (the backward pass of a differentiable regrid).
//
// A conservative weight is the area of the overlap of input cell i and
// output cell o divided by the area of input cell i (times weights_input[i]):
// the upstream computes it as a sum of contour pieces in its sweep
// (regridding/_weights/_weights_conservative_2d/_weights_conservative_2d.py:
// 752-830).  Its derivative with respect to the output vertices is taken
// here from the same overlap polygon built directly: the output quad is
// clipped against the (convex) input quad edge by edge, every vertex of the
// clipped polygon is typed as an output vertex, an input corner, or the
// crossing of output edge e with input edge f, and its position is computed
// from the original vertices.  The polygon area A = 1/2 sum cross(p_k, p_k+1)
// has dA/dp_k = 1/2 (y_k+1 - y_k-1, x_k-1 - x_k+1); a crossing
// p = a + t (b - a) with input edge c -> d carries it to the output vertices
// a and b as (1 - t) (G + (G.r) n) and t (G + (G.r) n), with r = b - a,
// s = d - c, n = (-s.y, s.x) / cross(r, s).
//
// Two kernels form the per-cell records of 8 coordinate derivatives:
//   * grad_edges: the usual rows.  Moving an output edge a -> b sweeps area at
//     its parts inside the input cell only, so with r = b - a,
//       dA/da = (r.y, -r.x) F_a,  F_a = integral of (1 - t) over those parts,
//       dA/db = (r.y, -r.x) F_b,  F_b = integral of t,
//     and the overlap polygon itself is not needed: only the parameters t at
//     which output edges enter and leave the cell;
//   * grad_polygons: every row when the weights recomputed from the polygons
//     are wanted, and (grad_polygons_listed) the rows grad_edges leaves.
// dL/dw_io = sum_d grad_out[d, o] * values[d, i] multiplies dw/dA.  A last
// kernel gives every output vertex the sum of its (up to four) cells' corner
// terms in a fixed order, so the gradient is the same bits on every run (no
// atomics).
#include <algorithm>

#include "common.cuh"

namespace rg {
namespace {

enum : unsigned { FLAG_NONCONVEX = 1u << 8, FLAG_DEGENERATE = 1u << 9 };

// A vertex of the clipped polygon, 40 bytes (two arrays of 12 per thread):
// a crossing keeps its parameter t and the reciprocal of its carriers'
// cross product, from which the gradient pass rebuilds the normal.
struct PV {
    double x, y;
    double t, inv;       // crossing data (kind 2): t along output edge e; 1 / cross(r, s)
    signed char ca, cb;  // carrier lines: 0..3 output edges, 4..7 input edges
    signed char kind;    // 0 output vertex (e), 1 input-only, 2 crossing (e, f)
    signed char e;
};

// float or double values as double (float: exactly, on the integer pipe)
__device__ __forceinline__ double as_double(float v) { return widen(v); }
__device__ __forceinline__ double as_double(double v) { return v; }

__device__ __forceinline__ double cross2(double ax, double ay, double bx, double by) { return ax * by - ay * bx; }

struct Quad {
    double x[4], y[4];
};

__device__ __forceinline__ void load_quad(const double* X, const double* Y, int64_t ny, int64_t i, int64_t j,
                                          Quad& q) {
    // vertex order (i, j), (i+1, j), (i+1, j+1), (i, j+1); edge k runs from
    // vertex k to vertex k+1
    const int64_t v0 = i * ny + j, v1 = (i + 1) * ny + j, v2 = (i + 1) * ny + j + 1, v3 = i * ny + j + 1;
    q.x[0] = __ldg(X + v0), q.y[0] = __ldg(Y + v0);
    q.x[1] = __ldg(X + v1), q.y[1] = __ldg(Y + v1);
    q.x[2] = __ldg(X + v2), q.y[2] = __ldg(Y + v2);
    q.x[3] = __ldg(X + v3), q.y[3] = __ldg(Y + v3);
}

__device__ __forceinline__ double quad_area2(const Quad& q) {
    return cross2(q.x[2] - q.x[0], q.y[2] - q.y[0], q.x[3] - q.x[1], q.y[3] - q.y[1]);
}

__device__ __forceinline__ bool convex(const Quad& q, double orient) {
    for (int k = 0; k < 4; k++) {
        const int a = k, b = (k + 1) & 3, c = (k + 2) & 3;
        if (orient * cross2(q.x[b] - q.x[a], q.y[b] - q.y[a], q.x[c] - q.x[b], q.y[c] - q.y[b]) < 0) return false;
    }
    return true;
}

// the carrier line shared by two consecutive polygon vertices
__device__ __forceinline__ int common_carrier(const PV& p, const PV& q, bool* ok) {
    if (p.ca == q.ca || p.ca == q.cb) return p.ca;
    if (p.cb == q.ca || p.cb == q.cb) return p.cb;
    *ok = false;
    return p.cb;
}

// crossing of carrier line L (output edge L, or input edge L - 4) with input edge f
__device__ PV crossing(const Quad& O, const Quad& C, int L, int f, bool* ok) {
    PV v;
    const double cx = C.x[f], cy = C.y[f];
    const double sx = C.x[(f + 1) & 3] - cx, sy = C.y[(f + 1) & 3] - cy;
    double ax, ay, rx, ry;
    if (L < 4) {
        ax = O.x[L], ay = O.y[L];
        rx = O.x[(L + 1) & 3] - ax, ry = O.y[(L + 1) & 3] - ay;
    } else {
        const int g = L - 4;
        ax = C.x[g], ay = C.y[g];
        rx = C.x[(g + 1) & 3] - ax, ry = C.y[(g + 1) & 3] - ay;
    }
    const double den = cross2(rx, ry, sx, sy);
    double t = 0, inv = 0;
    if (den != 0) {
        inv = 1.0 / den;  // one division serves t and (at the gradient) the normal
        t = cross2(cx - ax, cy - ay, sx, sy) * inv;
    } else {
        *ok = false;
    }
    v.x = ax + t * rx;
    v.y = ay + t * ry;
    v.ca = (signed char)L;
    v.cb = (signed char)(4 + f);
    if (L < 4) {
        v.kind = 2;
        v.e = (signed char)L;
        v.t = t;
        v.inv = inv;
    } else {
        v.kind = 1;
        v.e = -1;
        v.t = v.inv = 0;
    }
    return v;
}

template <typename T>
struct AdjointArgs {
    const int64_t* row_ptr;
    const int32_t* col;
    const double* val;
    int64_t n_in, n_out;
    const double *xi, *yi;
    int64_t nyi;
    const double *xo, *yo;
    int64_t nyo;
    const double* area_in;
    const double* w_in;   // nullable
    const double* scale;  // w_in / area_in of every input cell
    const T* values;
    const T* gout;
    int64_t stack;
    double* corner;   // 8 per output cell: its corners' x, then y derivatives
    double* w_check;  // nullable
    unsigned* flags;
};

// Adds to (ax, ay) the corner derivatives of output cell o from the clipped
// polygons of its entries first, first + step, ...
template <typename T>
__device__ void polygon_entries(const AdjointArgs<T>& A, int64_t o, int first, int step, double* ax, double* ay) {
    const int64_t* __restrict__ row_ptr = A.row_ptr;
    const int32_t* __restrict__ col = A.col;
    const double* __restrict__ val = A.val;
    const T* __restrict__ values = A.values;
    const T* __restrict__ gout = A.gout;
    const double* __restrict__ area_in = A.area_in;
    const double* __restrict__ w_in = A.w_in;
    const double *xi = A.xi, *yi = A.yi, *xo = A.xo, *yo = A.yo;
    const int64_t n_in = A.n_in, n_out = A.n_out, stack = A.stack, nyi = A.nyi, nyo = A.nyo;
    double* w_check = A.w_check;
    unsigned* flags = A.flags;
    const int64_t ncyo = nyo - 1, ncyi = nyi - 1;
    const int64_t io = o / ncyo, jo = o - io * ncyo;
    Quad O;
    load_quad(xo, yo, nyo, io, jo, O);
    for (int64_t k = row_ptr[o] + first; k < row_ptr[o + 1]; k += step) {
        const int64_t i = col[k];
        double G = 0;
        for (int64_t d = 0; d < stack; d++) G = fma(as_double(gout[d * n_out + o]), as_double(values[d * n_in + i]), G);
        if (G == 0 && w_check == nullptr) continue;
        const int64_t ii = i / ncyi, ji = i - ii * ncyi;
        Quad C;
        load_quad(xi, yi, nyi, ii, ji, C);
        const double orient = quad_area2(C) >= 0 ? 1.0 : -1.0;
        if (!convex(C, orient)) {
            atomicOr(flags, FLAG_NONCONVEX);
            continue;
        }
        // Sutherland-Hodgman: the output quad clipped by the 4 input edges
        PV poly[2][12];
        int m = 4;
        for (int v = 0; v < 4; v++) {
            PV& p = poly[0][v];
            p.x = O.x[v];
            p.y = O.y[v];
            p.ca = (signed char)((v + 3) & 3);
            p.cb = (signed char)v;
            p.kind = 0;
            p.e = (signed char)v;
            p.t = p.inv = 0;
        }
        int cur = 0;
        bool ok = true;
        for (int f = 0; f < 4 && m > 0; f++) {
            const double cx = C.x[f], cy = C.y[f];
            const double sx = C.x[(f + 1) & 3] - cx, sy = C.y[(f + 1) & 3] - cy;
            int n = 0;
            for (int v = 0; v < m; v++) {
                const PV& P = poly[cur][v];
                const PV& Q = poly[cur][(v + 1) % m];
                const bool pin = orient * cross2(sx, sy, P.x - cx, P.y - cy) >= 0;
                const bool qin = orient * cross2(sx, sy, Q.x - cx, Q.y - cy) >= 0;
                if (pin != qin && n < 12) poly[cur ^ 1][n++] = crossing(O, C, common_carrier(P, Q, &ok), f, &ok);
                if (qin && n < 12) poly[cur ^ 1][n++] = Q;
            }
            cur ^= 1;
            m = n;
        }
        if (!ok) atomicOr(flags, FLAG_DEGENERATE);
        if (m < 3) {
            if (w_check) w_check[k] = 0;
            continue;
        }
        const PV* p = poly[cur];
        double A2 = 0;
        for (int v = 0; v < m; v++) {
            const PV& a = p[v];
            const PV& b = p[(v + 1) % m];
            A2 += cross2(a.x, a.y, b.x, b.y);
        }
        const double ain = area_in[i];
        const double win = w_in ? w_in[i] : 1.0;
        double ratio = 0.5 * A2 / ain * win;
        // the stored weight fixes the sign convention (orientation of the grids)
        const double sgn = (val[k] * ratio < 0) ? -1.0 : 1.0;
        if (w_check) w_check[k] = sgn * ratio;
        if (G == 0) continue;
        const double c = G * sgn * win / ain;  // dL/dA
        for (int v = 0; v < m; v++) {
            const PV& q = p[v];
            if (q.kind == 1) continue;
            const PV& nx = p[(v + 1) % m];
            const PV& pv = p[(v + m - 1) % m];
            const double Gx = 0.5 * (nx.y - pv.y) * c, Gy = 0.5 * (pv.x - nx.x) * c;
            if (q.kind == 0) {
                ax[q.e] += Gx;
                ay[q.e] += Gy;
            } else {
                // the crossing of output edge e (r = b - a) with input edge f
                // (s): n = (-s.y, s.x) / cross(r, s)
                const int e0 = q.e, e1 = (q.e + 1) & 3, f0 = q.cb - 4, f1 = (q.cb - 3) & 3;
                const double rx = O.x[e1] - O.x[e0], ry = O.y[e1] - O.y[e0];
                const double nx = -(C.y[f1] - C.y[f0]) * q.inv, ny = (C.x[f1] - C.x[f0]) * q.inv;
                const double gr = Gx * rx + Gy * ry;
                const double hx = Gx + gr * nx, hy = Gy + gr * ny;
                const int a = q.e, b = (q.e + 1) & 3;
                ax[a] += (1 - q.t) * hx;
                ay[a] += (1 - q.t) * hy;
                ax[b] += q.t * hx;
                ay[b] += q.t * hy;
            }
        }
    }
}

// One thread per output cell.
template <typename T>
__global__ void __launch_bounds__(128) grad_polygons(const AdjointArgs<T> A) {
    const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= A.n_out) return;
    double ax[4] = {0, 0, 0, 0}, ay[4] = {0, 0, 0, 0};
    polygon_entries(A, o, 0, 1, ax, ay);
    double* rec = A.corner + o * 8;
    for (int v = 0; v < 4; v++) {
        rec[v] = ax[v];
        rec[4 + v] = ay[v];
    }
}

// The listed output cells, 8 lanes each: they are few, so the time is that of
// one lane's chain of polygons (a cell's 5 entries in one lane took 400 us).
template <typename T>
__global__ void __launch_bounds__(32)
    grad_polygons_listed(const AdjointArgs<T> A, const int32_t* __restrict__ rows, const unsigned* __restrict__ n_rows) {
    const int64_t total = *n_rows;
    const int lane = threadIdx.x & 7;
    for (int64_t q = blockIdx.x * 4; q < total; q += (int64_t)gridDim.x * 4) {
        const int64_t mine = q + (threadIdx.x >> 3);
        double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (mine < total) polygon_entries(A, (int64_t)rows[mine], lane, 8, a, a + 4);
        __syncwarp();
#pragma unroll
        for (int v = 0; v < 8; v++)
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) a[v] += __shfl_xor_sync(0xffffffffu, a[v], d);
        if (mine < total) {
            double own = a[0];
#pragma unroll
            for (int v = 1; v < 8; v++) own = lane == v ? a[v] : own;
            A.corner[(int64_t)rows[mine] * 8 + lane] = own;
        }
    }
}

// scale[i] = w_in[i] / area[i]: what turns an overlap area into a weight.
__global__ void area_scale(const double* __restrict__ area, const double* __restrict__ w_in, int64_t n,
                           double* __restrict__ scale) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        scale[i] = (w_in ? w_in[i] : 1.0) / area[i];
}

// v truncated to float32 from its bits, |v - f| < 2^-23 |v| (no FP64
// instruction).  Magnitudes below 2^-126 give 0; 2^128 and more, infinities
// and NaN give NaN, which no certain sign survives.
__device__ __forceinline__ float trunc_or_nan(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned ah = hi & 0x7fffffffu;
    const unsigned f = (hi & 0x80000000u) | ((ah - 0x38000000u) << 3) | (lo >> 29);
    return ah >= 0x47f00000u ? __int_as_float(0x7fffffff) : ah < 0x38100000u ? 0.f : __uint_as_float(f);
}

// ---------------------------------------------------------------------------
// The usual rows.  GB300 issues 2 FP64 operations per clock per SM, 1/64 of
// its FP32 rate, so the kernel decides where edges meet in float32, with an
// error bound, and spends FP64 on the crossings alone.
//
// A warp takes 8 output cells, its lanes their entries 32 at a time.  Per
// entry the 16 orientations of output vertices against input edges and the
// 16 of input vertices against output edges are evaluated in float32 from
// coordinates relative to the output cell's first vertex (differences taken
// in FP64, then truncated).  Output edge e meets input edge f of the convex
// cell exactly where the ends of each lie on opposite sides of the other; an
// edge whose end is inside all four input edges leaves at t = 1.  With M the
// largest magnitude among the pair's local coordinates, a float32 difference
// is within 2^-21 M of the exact one and at most 2 M, so an orientation
// s.x d.y - s.y d.x is off by less than
//   8 2^-21 M^2 (the differences) + 2 2^-42 M^2 + 12 2^-24 M^2 (its roundings),
// under 2^-17 M^2 = E.  An orientation within E of zero is taken in FP64.  A
// cell is left to the polygons when one is not certain there either (a
// vertex on an edge's line), when either quad is not certainly convex, or
// when an overlap is below 2^-47 X^2, X the largest coordinate (the sign
// convention, val against the polygon's area, hangs on that area there, which
// the polygons' absolute coordinates round by up to 24 2^-53 X^2).
//
// The crossings of a warp's 32 entries, about two per entry, are queued and
// taken one per lane, so the FP64 work (22 operations and a division each)
// runs on full warps; each entry's enter and leave values of F_a and F_b meet
// in shared memory, and lane 4 r + e adds those of edge e of cell r in stored
// order.  FP64 issue and the latency of its chains bound the kernel.
// ---------------------------------------------------------------------------

constexpr int EDGE_ROWS = 8;   // output cells of a warp
constexpr int EDGE_WARPS = 4;  // warps of a block

struct EdgeWarp {
    double cx[4][32], cy[4][32];                  // input quads of the entries, local
    double ox[EDGE_ROWS][4], oy[EDGE_ROWS][4];    // output quads, local to their first vertex
    double fa[2][4][32], fb[2][4][32];            // enter, leave values of F_a and F_b
    double dldw[32];                              // dL/dA of the entries
    int64_t rp[EDGE_ROWS + 1];
    unsigned short queue[32 * 8];                 // lane | e << 5 | f << 7 | leaves << 9
    unsigned char row[32], touched[32];           // the entry's cell; its edges with parts inside
    int8_t orient[EDGE_ROWS];                     // of the output quad; 0: not certainly convex
    unsigned hard;                                // cells left to grad_polygons
};

template <typename T>
__global__ void __launch_bounds__(32 * EDGE_WARPS)
    grad_edges(const AdjointArgs<T> A, int32_t* __restrict__ rows, unsigned* __restrict__ n_rows) {
    __shared__ EdgeWarp shared[EDGE_WARPS];
    EdgeWarp& S = shared[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int64_t o0 = (blockIdx.x * (int64_t)EDGE_WARPS + (threadIdx.x >> 5)) * EDGE_ROWS;
    if (o0 >= A.n_out) return;  // whole warps
    const int r_mine = lane >> 2, e_mine = lane & 3, next = (lane & ~3) | ((lane + 1) & 3);
    const int64_t ncyo = A.nyo - 1, ncyi = A.nyi - 1;
    // lane 4 r + e: vertex e of cell r (a cell past the end repeats the last one)
    const int64_t o = o0 + r_mine < A.n_out ? o0 + r_mine : A.n_out - 1;
    double edge_x, edge_y;  // this lane's output edge e -> e + 1
    {
        const int64_t i = o / ncyo, j = o - i * ncyo;
        const int64_t v = (i + (e_mine == 1 || e_mine == 2)) * A.nyo + j + (e_mine >= 2);
        const double x = __ldg(A.xo + v), y = __ldg(A.yo + v);
        const double lx = x - __shfl_sync(0xffffffffu, x, lane & ~3);
        const double ly = y - __shfl_sync(0xffffffffu, y, lane & ~3);
        S.ox[r_mine][e_mine] = lx;
        S.oy[r_mine][e_mine] = ly;
        edge_x = __shfl_sync(0xffffffffu, lx, next) - lx;
        edge_y = __shfl_sync(0xffffffffu, ly, next) - ly;
        // orientation at vertex e + 1
        const float fx = trunc_or_nan(lx), fy = trunc_or_nan(ly);
        const float gx = __shfl_sync(0xffffffffu, fx, next), gy = __shfl_sync(0xffffffffu, fy, next);
        const float hx = __shfl_sync(0xffffffffu, gx, next), hy = __shfl_sync(0xffffffffu, gy, next);
        float M = fmaxf(fabsf(fx), fabsf(fy));
        M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 1));
        M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 2));
        const float c = (gx - fx) * (hy - gy) - (gy - fy) * (hx - gx);
        const bool sure = fabsf(c) > M * M * 7.62939453e-6f && M > 9.094947e-13f && M < 1.0995116e12f;  // 2^-17, 2^-40, 2^40
        const unsigned up = __ballot_sync(0xffffffffu, sure && c > 0.f) >> (lane & ~3) & 15u;
        const unsigned down = __ballot_sync(0xffffffffu, sure && c < 0.f) >> (lane & ~3) & 15u;
        if (e_mine == 0) S.orient[r_mine] = up == 15u ? 1 : down == 15u ? -1 : 0;
    }
    if (lane <= EDGE_ROWS) S.rp[lane] = A.row_ptr[o0 + lane < A.n_out ? o0 + lane : A.n_out];
    if (lane == 0) S.hard = 0u;
    __syncwarp();
    const int64_t k_end = S.rp[EDGE_ROWS];
    double sum_a = 0.0, sum_b = 0.0;  // of edge e of cell r: sum dL/dA F_a, sum dL/dA F_b
    for (int64_t k0 = S.rp[0]; k0 < k_end; k0 += 32) {
        const int64_t k = k0 + lane;
        unsigned meet = 0u, leave = 0u;  // bits e * 4 + f: crossing, and it leaves the cell
        unsigned ends = 0u;              // bits e: the edge's end is inside
        if (k < k_end) {
            int r = 0;
            for (int q = 1; q < EDGE_ROWS; q++) r += S.rp[q] <= k;
            S.row[lane] = (unsigned char)r;
            const int64_t out = o0 + r, i = A.col[k];
            double G = 0;
            for (int64_t d = 0; d < A.stack; d++)
                G = fma(as_double(A.gout[d * A.n_out + out]), as_double(A.values[d * A.n_in + i]), G);
            if (G != 0) {
                const int64_t ii = i / ncyi, ji = i - ii * ncyi;
                const int64_t b = (out / ncyo) * A.nyo + out % ncyo;
                const double x0 = __ldg(A.xo + b), y0 = __ldg(A.yo + b);
                Quad C;
                load_quad(A.xi, A.yi, A.nyi, ii, ji, C);
                float px[4], py[4], qx[4], qy[4];  // output and input vertices
                float M = 0.f;
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const double lx = C.x[v] - x0, ly = C.y[v] - y0;
                    S.cx[v][lane] = lx;
                    S.cy[v][lane] = ly;
                    qx[v] = trunc_or_nan(lx);
                    qy[v] = trunc_or_nan(ly);
                    px[v] = trunc_or_nan(S.ox[r][v]);
                    py[v] = trunc_or_nan(S.oy[r][v]);
                    M = fmaxf(M, fmaxf(fmaxf(fabsf(qx[v]), fabsf(qy[v])), fmaxf(fabsf(px[v]), fabsf(py[v]))));
                }
                const float E = M * M * 7.62939453e-6f;  // 2^-17
                auto orientation = [](float sx, float sy, float dx, float dy) { return sx * dy - sy * dx; };
                unsigned turns = 0u;  // bits v: the input quad turns left there
                bool usual = M > 9.094947e-13f && M < 1.0995116e12f;
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const int g = (v + 1) & 3, h = (v + 2) & 3;
                    const float c = orientation(qx[g] - qx[v], qy[g] - qy[v], qx[h] - qx[g], qy[h] - qy[g]);
                    usual = usual && fabsf(c) > E;
                    turns |= (unsigned)(c > 0.f) << v;
                }
                // bits v * 4 + f: output v left of input f, and not certain;
                // bits e * 4 + v: input v left of output e, and not certain
                unsigned inside = 0u, inside_open = 0u, left = 0u, left_open = 0u;
#pragma unroll
                for (int a = 0; a < 4; a++) {
                    const int b1 = (a + 1) & 3;
                    const float sx = qx[b1] - qx[a], sy = qy[b1] - qy[a];
                    const float rx = px[b1] - px[a], ry = py[b1] - py[a];
#pragma unroll
                    for (int v = 0; v < 4; v++) {
                        const float ci = orientation(sx, sy, px[v] - qx[a], py[v] - qy[a]);
                        const float co = orientation(rx, ry, qx[v] - px[a], qy[v] - py[a]);
                        inside |= (unsigned)(ci > 0.f) << (v * 4 + a);
                        inside_open |= (unsigned)!(fabsf(ci) > E) << (v * 4 + a);
                        left |= (unsigned)(co > 0.f) << (a * 4 + v);
                        left_open |= (unsigned)!(fabsf(co) > E) << (a * 4 + v);
                    }
                }
                // the open ones in FP64, off by under 2^-46 M^2 (as above
                // with 2^-53 for 2^-24)
                const double E64 = (double)(M * M) * 1.4210854715202004e-14;
                auto settle = [&](unsigned open, unsigned& bits, const double* px, const double* py, int ps,
                                  const double* lx, const double* ly, int ls, bool line_low) {
                    for (; open; open &= open - 1u) {
                        const int bit = __ffs(open) - 1;
                        const int line = line_low ? bit & 3 : bit >> 2, v = line_low ? bit >> 2 : bit & 3;
                        const int l1 = (line + 1) & 3;
                        const double ax = lx[line * ls], ay = ly[line * ls];
                        const double c = cross2(lx[l1 * ls] - ax, ly[l1 * ls] - ay, px[v * ps] - ax, py[v * ps] - ay);
                        usual = usual && fabs(c) > E64;
                        bits = (bits & ~(1u << bit)) | (unsigned)(c > 0) << bit;
                    }
                };
                settle(inside_open, inside, S.ox[r], S.oy[r], 1, &S.cx[0][lane], &S.cy[0][lane], 32, true);
                settle(left_open, left, &S.cx[0][lane], &S.cy[0][lane], 32, S.ox[r], S.oy[r], 1, false);
                if (turns == 0u) inside = ~inside & 0xffffu;  // clockwise input cell
                const int orient = S.orient[r];
                const double w = A.val[k], scale = A.scale[i];
                const float X = fmaxf(fabsf(trunc_or_nan(x0)), fabsf(trunc_or_nan(y0))) + M;
                usual = usual && (turns == 0u || turns == 15u) && orient != 0 &&
                        fabsf((float)w) >= 7.1054274e-15f * X * X * fabsf((float)scale);  // 2^-47
                if (!usual) {
                    atomicOr(&S.hard, 1u << r);
                } else {
                    const unsigned sign = (unsigned)((__double2hiint(w) ^ __double2hiint(scale)) >> 31) ^
                                          (unsigned)(orient >> 31);
                    const double c = G * scale;
                    S.dldw[lane] = sign & 1u ? -c : c;
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const unsigned ia = inside >> (e * 4) & 15u, ib = inside >> (((e + 1) & 3) * 4) & 15u;
                        const unsigned le = left >> (e * 4) & 15u;
                        const unsigned split = le ^ ((le >> 1) | (le << 3 & 8u));  // bit f: input edge f's ends on both sides
                        meet |= ((ia ^ ib) & split) << (e * 4);
                        leave |= (ia & ~ib & split) << (e * 4);
                        ends |= (unsigned)(ib == 15u) << e;
                    }
                }
            }
        }
        unsigned touched = ends;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const bool out = (ends >> e) & 1u;  // leaves at t = 1: F_a = F_b = 1/2
            S.fa[0][e][lane] = 0.0;
            S.fb[0][e][lane] = 0.0;
            S.fa[1][e][lane] = out ? 0.5 : 0.0;
            S.fb[1][e][lane] = out ? 0.5 : 0.0;
            touched |= (unsigned)((meet >> (e * 4) & 15u) != 0u) << e;
        }
        S.touched[lane] = (unsigned char)touched;
        // queue the crossings: a convex cell has at most 8
        int at = __popc(meet);
        const int mine = at;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, at, d);
            if (lane >= d) at += up;
        }
        const int total = __shfl_sync(0xffffffffu, at, 31);
        at -= mine;
        for (unsigned left = meet; left; left &= left - 1u, at++) {
            const int bit = __ffs(left) - 1;
            S.queue[at] = (unsigned short)(lane | (bit >> 2) << 5 | (bit & 3) << 7 | (leave >> bit & 1u) << 9);
        }
        __syncwarp();
        for (int q = lane; q < total; q += 32) {
            const unsigned code = S.queue[q];
            const int en = code & 31, e = code >> 5 & 3, f = code >> 7 & 3, out = code >> 9;
            const int r = S.row[en], e1 = (e + 1) & 3, f1 = (f + 1) & 3;
            const double ax = S.ox[r][e], ay = S.oy[r][e];
            const double rx = S.ox[r][e1] - ax, ry = S.oy[r][e1] - ay;
            const double cx = S.cx[f][en], cy = S.cy[f][en];
            const double sx = S.cx[f1][en] - cx, sy = S.cy[f1][en] - cy;
            const double t = cross2(cx - ax, cy - ay, sx, sy) / cross2(rx, ry, sx, sy);
            const double half = 0.5 * t * t;
            S.fa[out][e][en] = t - half;
            S.fb[out][e][en] = half;
        }
        __syncwarp();
        // this lane's edge over its cell's entries of the batch
        const int64_t a = S.rp[r_mine] > k0 ? S.rp[r_mine] : k0;
        const int64_t b = S.rp[r_mine + 1] < k0 + 32 ? S.rp[r_mine + 1] : k0 + 32;
        for (int64_t q = a; q < b; q++) {
            const int en = (int)(q - k0);
            if (S.touched[en] >> e_mine & 1u) {
                const double c = S.dldw[en];
                sum_a = fma(c, S.fa[1][e_mine][en] - S.fa[0][e_mine][en], sum_a);
                sum_b = fma(c, S.fb[1][e_mine][en] - S.fb[0][e_mine][en], sum_b);
            }
        }
        __syncwarp();
    }
    // corner e: edge e at its start, edge e - 1 at its end
    const int prev = (lane & ~3) | ((lane + 3) & 3);
    const double gx = edge_y * sum_a + __shfl_sync(0xffffffffu, edge_y * sum_b, prev);
    const double gy = -(edge_x * sum_a + __shfl_sync(0xffffffffu, edge_x * sum_b, prev));
    if (o0 + r_mine < A.n_out) {
        double* rec = A.corner + (o0 + r_mine) * 8;
        rec[e_mine] = gx;
        rec[4 + e_mine] = gy;
        if (e_mine == 0 && (S.hard >> r_mine & 1u)) rows[atomicAdd(n_rows, 1u)] = (int32_t)(o0 + r_mine);
    }
}

// Records of all output cells (stream ordered).
template <typename T>
int adjoint_records(const AdjointArgs<T>& A, int32_t* rows, unsigned* n_rows, cudaStream_t s) {
    if (A.w_check) {
        grad_polygons<T><<<grid_for(A.n_out, 128), 128, 0, s>>>(A);
    } else {
        grad_edges<T><<<grid_for(A.n_out, EDGE_WARPS * EDGE_ROWS), 32 * EDGE_WARPS, 0, s>>>(A, rows, n_rows);
        grad_polygons_listed<T><<<std::min(grid_for(A.n_out, 4), 152u * 16u), 32, 0, s>>>(A, rows, n_rows);
    }
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

// Gradient of output vertex (a, b): corner 0 of cell (a, b), corner 1 of
// cell (a - 1, b), corner 2 of cell (a - 1, b - 1) and corner 3 of cell
// (a, b - 1), those that exist, added in that order.
__global__ void __launch_bounds__(256)
    vertex_sum(const double* __restrict__ corner, int64_t nxo, int64_t nyo, double* __restrict__ gx,
               double* __restrict__ gy) {
    const int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (v >= nxo * nyo) return;
    const int64_t a = v / nyo, b = v - a * nyo, ncy = nyo - 1;
    double sx = 0.0, sy = 0.0;
    const int64_t ci[4] = {a, a - 1, a - 1, a};
    const int64_t cj[4] = {b, b, b - 1, b - 1};
    for (int c = 0; c < 4; c++) {
        if (ci[c] < 0 || ci[c] >= nxo - 1 || cj[c] < 0 || cj[c] >= ncy) continue;
        const double* rec = corner + (ci[c] * ncy + cj[c]) * 8;
        sx += rec[c];
        sy += rec[4 + c];
    }
    gx[v] = sx;
    gy[v] = sy;
}

}  // namespace

int cell_area_2d(const double* x, const double* y, int64_t nx, int64_t ny, double* area, cudaStream_t s);

}  // namespace rg

extern "C" int rg_conservative_2d_grad_output(rg_weights w, const double* d_xi, const double* d_yi, int64_t nxi,
                                              int64_t nyi, const double* d_xo, const double* d_yo, int64_t nxo,
                                              int64_t nyo, const double* d_w_in, const void* d_values,
                                              const void* d_grad_out, int dtype, int64_t stack, double* d_grad_xo,
                                              double* d_grad_yo, double* d_w_check, rg_stream_t stream) {
    rg::NvtxRange nvtx_range("rg_conservative_2d_grad_output");
    using namespace rg;
    RG_CHECK(w, RG_ERR_ARG, "rg_conservative_2d_grad_output: NULL handle");
    RG_CHECK(nxi >= 2 && nyi >= 2 && nxo >= 2 && nyo >= 2, RG_ERR_ARG,
             "rg_conservative_2d_grad_output: grids need at least 2 vertices per axis");
    RG_CHECK(w->n_in == (nxi - 1) * (nyi - 1) && w->n_out == (nxo - 1) * (nyo - 1), RG_ERR_ARG,
             "rg_conservative_2d_grad_output: grids do not match the weights (%lld -> %lld cells)",
             (long long)w->n_in, (long long)w->n_out);
    RG_CHECK(dtype == RG_F32 || dtype == RG_F64, RG_ERR_ARG, "rg_conservative_2d_grad_output: bad dtype");
    RG_CHECK(stack >= 0, RG_ERR_ARG, "rg_conservative_2d_grad_output: negative stack");
    cudaStream_t s = (cudaStream_t)stream;
    const int64_t nv = nxo * nyo;
    if (w->n_out == 0 || w->nnz == 0) {
        RG_CUDA(cudaMemsetAsync(d_grad_xo, 0, sizeof(double) * nv, s));
        RG_CUDA(cudaMemsetAsync(d_grad_yo, 0, sizeof(double) * nv, s));
        return RG_OK;
    }
    double *area = nullptr, *scale = nullptr;
    double* corner = nullptr;
    unsigned* flags = nullptr;  // [0] conditions met, [1] listed cells
    int32_t* rows = nullptr;
    int st = RG_OK;
    do {
        if ((st = dalloc(&area, (size_t)w->n_in, s))) break;
        if ((st = dalloc(&scale, (size_t)w->n_in, s))) break;
        if ((st = dalloc(&corner, (size_t)w->n_out * 8, s))) break;
        if ((st = dalloc(&rows, (size_t)w->n_out, s))) break;
        if ((st = dalloc(&flags, 2, s))) break;
        cudaMemsetAsync(flags, 0, 2 * sizeof(unsigned), s);
        if ((st = cell_area_2d(d_xi, d_yi, nxi, nyi, area, s))) break;
        area_scale<<<std::min(grid_for(w->n_in, 256), 8192u), 256, 0, s>>>(area, d_w_in, w->n_in, scale);
        auto records = [&](auto zero) {
            using T = decltype(zero);
            return adjoint_records<T>({w->row_ptr, w->col, w->val, w->n_in, w->n_out, d_xi, d_yi, nyi, d_xo, d_yo, nyo,
                                       area, d_w_in, scale, (const T*)d_values, (const T*)d_grad_out, stack, corner,
                                       d_w_check, flags},
                                      rows, flags + 1, s);
        };
        if ((st = dtype == RG_F32 ? records(0.f) : records(0.0))) break;
        vertex_sum<<<grid_for(nv, 256), 256, 0, s>>>(corner, nxo, nyo, d_grad_xo, d_grad_yo);
        unsigned fl = 0;
        cudaMemcpyAsync(&fl, flags, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
        cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error("rg_conservative_2d_grad_output: %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
            break;
        }
        if (fl & FLAG_NONCONVEX) {
            set_error("rg_conservative_2d_grad_output: an input cell is not convex (the overlap clipping "
                      "needs convex input cells)");
            st = RG_ERR_UNSUPPORTED;
        } else if (fl & FLAG_DEGENERATE) {
            set_error("rg_conservative_2d_grad_output: degenerate overlap (parallel or coincident edges)");
            st = RG_ERR_UNSUPPORTED;
        }
    } while (0);
    dfree(area, s);
    dfree(scale, s);
    dfree(corner, s);
    dfree(rows, s);
    dfree(flags, s);
    return st;
}
