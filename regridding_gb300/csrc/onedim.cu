// 1D kernels: find_indices (brute and searchsorted), multilinear weights and
// conservative 1D weights over batches of rows.
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace rg {
namespace {

// numpy.searchsorted(a, v, side="left") on an ascending row: the first k with
// a[k] >= v in numpy's float order (NaN after every number).
__device__ __forceinline__ int64_t lower_bound_np(const double* a, int64_t n, double v) {
    int64_t lo = 0, hi = n;
    bool vnan = isnan(v);
    while (lo < hi) {
        int64_t mid = lo + ((hi - lo) >> 1);
        double am = __ldg(a + mid);
        bool lt = (am < v) || (vnan && !isnan(am));
        if (lt) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// _find_indices_searchsorted_1d post-processing: _find_indices_searchsorted.py:47-58
__device__ __forceinline__ int64_t searchsorted_cell(const double* a, int64_t m, double p,
                                                     int64_t fill) {
    int64_t r = lower_bound_np(a, m, p) - 1;
    if (p == __ldg(a)) r = 0;
    else if (r < 0) r = fill;
    else if (r > m - 2) r = fill;
    return r;
}

// Rows that are non-decreasing (and NaN free) answer the brute search with a
// binary search: for them the first m with a[m] <= p <= a[m+1] is exactly the
// searchsorted cell.  Other rows are scanned linearly.
__global__ void row_sorted_kernel(const double* x, int64_t stride, int64_t m, int64_t nrows,
                                  uint8_t* sorted) {
    int lane = threadIdx.x & 31;
    int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (r >= nrows) return;
    const double* a = x + r * stride;
    bool ok = true;
    for (int64_t k = lane; k + 1 < m; k += 32) ok &= (a[k] <= a[k + 1]);
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) sorted[r] = ok;
}

__global__ void find_indices_kernel(const double* __restrict__ xin, int64_t in_stride, int64_t m,
                                    const double* __restrict__ xout, int64_t out_stride, int64_t n,
                                    int64_t nd, int method, int64_t fill,
                                    const uint8_t* __restrict__ sorted, int64_t* __restrict__ res) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nd * n;
         k += (int64_t)gridDim.x * blockDim.x) {
        int64_t d = k / n, i = k % n;
        const double* a = xin + d * in_stride;
        double p = xout[d * out_stride + i];
        int64_t r;
        if (method == 1) {
            r = searchsorted_cell(a, m, p, fill);
        } else if (m < 2) {
            r = fill;
        } else if (sorted[in_stride ? d : 0]) {
            r = searchsorted_cell(a, m, p, fill);
        } else {
            // _find_indices_brute_1d: _find_indices_brute.py:42-49
            r = fill;
            for (int64_t q = 0; q < m - 1; q++) {
                if (a[q] <= p && p <= a[q + 1]) {
                    r = q;
                    break;
                }
            }
        }
        res[k] = r;
    }
}

// _weights_from_indices_multilinear (_weights_multilinear.py:101-126) and
// _weights_from_indices_multilinear_1d (:169-202): raw entries 2i, 2i+1 of
// every row, plus the bucket (row, input index) and the in-bucket key
// (output index) used to put each row in the saved (input, output) order.
__global__ void multilinear_kernel(const double* __restrict__ xin, int64_t in_stride, int64_t m,
                                   const double* __restrict__ xout,
                                   const double* __restrict__ xsearch, int64_t out_stride, int64_t n,
                                   int64_t nd, const double* __restrict__ w_in, int64_t w_stride,
                                   int bounds, int32_t* __restrict__ bucket,
                                   int64_t* __restrict__ skey, double* __restrict__ raw_val,
                                   unsigned long long* __restrict__ n_outside) {
    const int64_t index_max = m - 2;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nd * n;
         k += (int64_t)gridDim.x * blockDim.x) {
        int64_t d = k / n, i = k % n;
        const double* a = xin + d * in_stride;
        double x = xout[d * out_stride + i];
        int64_t index = searchsorted_cell(a, m, xsearch ? xsearch[d * out_stride + i] : x, INT64_MAX);
        bool outside = (index < 0) || (index > index_max);
        if (outside && n_outside) atomicAdd(n_outside, 1ull);
        bool below = x < __ldg(a);
        int64_t i0 = below ? 0 : (index < 0 ? 0 : (index > index_max ? index_max : index));
        int64_t i1 = i0 + 1;
        double x0 = __ldg(a + i0), x1 = __ldg(a + i1);
        double w1 = ddiv(dsub(x, x0), dsub(x1, x0));
        double w0 = dsub(1.0, w1);
        if (w_in) {
            w0 = dmul(w0, w_in[d * w_stride + i0]);
            w1 = dmul(w1, w_in[d * w_stride + i1]);
        }
        if (bounds == RG_BOUNDS_NAN && outside) {
            w0 = NAN;
            w1 = NAN;
        }
        int64_t e = d * 2 * n + 2 * i;
        bucket[e] = (int32_t)(d * (m) + i0);
        bucket[e + 1] = (int32_t)(d * (m) + i1);
        skey[e] = i;
        skey[e + 1] = i;
        raw_val[e] = w0;
        raw_val[e + 1] = w1;
    }
}

__global__ void gather_multilinear(const uint32_t* __restrict__ perm, const int32_t* __restrict__ bucket,
                                   const int64_t* __restrict__ skey, const double* __restrict__ raw_val,
                                   int64_t total, int64_t m, int64_t* __restrict__ ind_in,
                                   int64_t* __restrict__ ind_out, double* __restrict__ val) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total;
         k += (int64_t)gridDim.x * blockDim.x) {
        uint32_t e = perm[k];
        ind_in[k] = bucket[e] % m;
        ind_out[k] = skey[e];
        val[k] = raw_val[e];
    }
}

// One row of _weights_conservative_1d (_weights_conservative_1d.py:59-318).
// Grids are read through index maps instead of reversed copies.
struct Row1d {
    const double *in, *out;
    int64_t m, n;
    bool rev_in, rev_out;
    __device__ __forceinline__ Row1d(const double* a, const double* b, int64_t m, int64_t n)
        : in(a), out(b), m(m), n(n), rev_in(!(a[0] < a[m - 1])), rev_out(!(b[0] < b[n - 1])) {}
    __device__ __forceinline__ double xs(int64_t k) const { return __ldg(in + (rev_in ? m - 1 - k : k)); }
    __device__ __forceinline__ double xt(int64_t k) const { return __ldg(out + (rev_out ? n - 1 - k : k)); }
    // weight of the piece p1..p2 of sweep cell isw, with the length of the
    // (possibly reversed) sweep grid's cell at its saved index (negative
    // indices wrap, as numpy indexing does)
    __device__ __forceinline__ double weight(double p1, double p2, int64_t isw, const double* w_in) const {
        const int64_t li = rev_in ? m - 2 - isw : isw;
        double ratio = ddiv(dsub(p2, p1), dsub(xs(li + 1), xs(li)));
        return w_in ? dmul(ratio, w_in[li]) : ratio;
    }
};

// first k in [0, n) with at(k) >= v (or > v), at() ascending
template <typename At>
__device__ __forceinline__ int64_t first_not_below(const At& at, int64_t n, double v) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (at(mid) < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
template <typename At>
__device__ __forceinline__ int64_t first_above(const At& at, int64_t n, double v) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (at(mid) <= v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The sweep of one row, entry by entry.
struct Sweep1d {
    int64_t isw = 0, ist = MAXSIZE;
    double p1;
    bool outside = true, ended = false;

    __device__ __forceinline__ Sweep1d(const Row1d& R) : p1(R.xs(0)) {
        const double left = R.xt(0), right = R.xt(R.n - 1);
        if (left == p1) {
            outside = false;
            ist = 0;
        } else if (left < p1 && p1 < right) {
            outside = false;
            int64_t l = 0, r = R.n;
            while (r - l > 1) {
                const int64_t mid = (l + r) / 2;
                if (R.xt(mid) > p1) r = mid;
                else l = mid;
            }
            ist = r - 1;
        }
    }
    __device__ __forceinline__ bool live(const Row1d& R) const { return !ended && isw < R.m - 1; }
    // One step; true when it made an entry, of cells sw and st from `from` to `to`.
    __device__ __forceinline__ bool step(const Row1d& R, int64_t* sw, int64_t* st, double* from, double* to) {
        double p2 = R.xs(isw + 1);
        *sw = isw;
        *st = ist;
        *from = p1;
        const bool entry = !outside;
        const double ps = R.xt(outside ? 0 : ist + 1);
        if (p1 < ps && ps < p2) {
            ist = outside ? 0 : ist + 1;
            p2 = ps;
        } else {
            if (ps == p2) ist = outside ? 0 : ist + 1;
            isw = isw + 1;
        }
        if (entry) ended = !(0 <= ist && ist < R.n - 1);
        else outside = !(ist < MAXSIZE);
        *to = p1 = p2;
        return entry;
    }
};

// The entries of one row by one thread, in the saved order.  Every entry moves
// on in the sweep grid or the static one and none moves back, so pairs are
// unique, entries of one input are neighbours, and the saved order (by input,
// then output) is the sweep's, reversed as a whole (reversed input: a sweep
// ahead counts the entries) and within the inputs (one of the grids reversed:
// each input's entries are turned round once they are written).
__device__ __noinline__ int64_t sweep_1d(const Row1d& R, const double* w_in, int64_t cap, int64_t* ind_in,
                                         int64_t* ind_out, double* val, unsigned* flags) {
    int64_t sw, st, total = 0, cnt = 0;
    double from, to;
    if (R.rev_in)
        for (Sweep1d ahead(R); ahead.live(R);) total += ahead.step(R, &sw, &st, &from, &to);
    const auto place = [&](int64_t k) { return R.rev_in ? total - 1 - k : k; };
    const bool turn = R.rev_in != R.rev_out;
    int64_t own = -1, first = 0;  // the current input and its first entry
    const auto turn_round = [&]() {
        int64_t a = place(first), b = place(cnt - 1);
        if (a > b) {
            const int64_t t = a;
            a = b;
            b = t;
        }
        for (; a < b; a++, b--) {
            const int64_t o = ind_out[a];
            const double v = val[a];
            ind_out[a] = ind_out[b];
            val[a] = val[b];
            ind_out[b] = o;
            val[b] = v;
        }
    };
    for (Sweep1d sweep(R); sweep.live(R);) {
        if (!sweep.step(R, &sw, &st, &from, &to)) continue;
        if (turn && sw != own) {
            if (cnt - first > 1) turn_round();
            own = sw;
            first = cnt;
        }
        const int64_t at = place(cnt);
        if (at >= cap) {
            atomicOr(flags, FLAG_CAPACITY);
            return 0;
        }
        ind_in[at] = R.rev_in ? ~sw : sw;
        ind_out[at] = R.rev_out ? ~st : st;
        val[at] = R.weight(from, to, sw, w_in);
        cnt++;
    }
    if (turn && cnt - first > 1) turn_round();
    return cnt;
}

// One block per row.  Where both grids rise strictly in sweep order, the sweep
// visits their vertices on the common range in order, a vertex of both once,
// and emits one entry from each to the next: a merge.  Every vertex finds its
// place by binary search: that of sweep vertex j is its rank among the sweep
// vertices plus the static ones before it that are no sweep vertices (before,
// in rank order), and so on for the static ones, so the entries are written
// where they are saved, with no sort.  The former thread per row, sort by
// buckets and thread per row for the merge spent 2.1 ms on 256 rows of 513 and
// 385 vertices (chains of a few hundred dependent steps); this takes 52 us.
// The first `few` rows that do not rise strictly are swept by the block's
// first thread, beside the other blocks; further ones are listed for
// conservative_1d_sweeps.  (10,000 such rows of 513 and 385 vertices one thread
// a block: 16 ms, now 1.7.)
constexpr int CONS_THREADS = 256;

__global__ void __launch_bounds__(CONS_THREADS)
    conservative_1d_rows(const double* __restrict__ xin, int64_t in_stride, int64_t m, const double* __restrict__ xout,
                         int64_t out_stride, int64_t n, int64_t nd, const double* __restrict__ w_in, int64_t w_stride,
                         int64_t cap, int64_t* __restrict__ ind_in, int64_t* __restrict__ ind_out,
                         double* __restrict__ val, int64_t* __restrict__ count, int* __restrict__ rank_all,
                         unsigned* flags, int32_t* __restrict__ list, unsigned* __restrict__ n_list, unsigned few) {
    extern __shared__ int rank_shared[];
    __shared__ int warp_sum[CONS_THREADS / 32];
    __shared__ int running;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int64_t d = blockIdx.x; d < nd; d += gridDim.x) {
        const Row1d R(xin + d * in_stride, xout + d * out_stride, m, n);
        const double* w_row = w_in ? w_in + d * w_stride : nullptr;
        int64_t* o_in = ind_in + d * cap;
        int64_t* o_out = ind_out + d * cap;
        double* o_val = val + d * cap;
        bool rises = true;
        for (int64_t k = t; k + 1 < m; k += CONS_THREADS) rises = rises && R.xs(k) < R.xs(k + 1);
        for (int64_t k = t; k + 1 < n; k += CONS_THREADS) rises = rises && R.xt(k) < R.xt(k + 1);
        if (!__syncthreads_and(rises)) {
            if (t == 0) {
                const unsigned at = atomicAdd(n_list, 1u);
                if (at < few) count[d] = sweep_1d(R, w_row, cap, o_in, o_out, o_val, flags);
                else list[at - few] = (int32_t)d;
            }
            continue;
        }
        const auto xs = [&](int64_t k) { return R.xs(k); };
        const auto xt = [&](int64_t k) { return R.xt(k); };
        // rank[k]: static vertices before k that are no sweep vertices
        int* rank = rank_all ? rank_all + blockIdx.x * (n + 1) : rank_shared;
        if (t == 0) running = 0;
        for (int64_t k0 = 0; k0 <= n; k0 += CONS_THREADS) {
            const int64_t k = k0 + t;
            int own = 0;
            if (k < n) {
                const double v = R.xt(k);
                const int64_t j = first_not_below(xs, m, v);
                own = !(j < m && R.xs(j) == v);
            }
            int incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            if (lane == 31) warp_sum[warp] = incl;
            __syncthreads();
            int before = running;
            for (int w = 0; w < warp; w++) before += warp_sum[w];
            if (k <= n) rank[k] = before + incl - own;
            __syncthreads();
            if (t == CONS_THREADS - 1) running = before + incl;
        }
        __syncthreads();
        // the common range: its vertices are places 0 .. entries
        const double a = fmax(R.xs(0), R.xt(0)), b = fmin(R.xs(m - 1), R.xt(n - 1));
        const int64_t ja = first_not_below(xs, m, a), ka = first_not_below(xt, n, a);
        const auto place_before = [&](int64_t j, int64_t k) { return j - ja + rank[k] - rank[ka]; };
        const int64_t entries = a < b ? place_before(first_not_below(xs, m, b), first_not_below(xt, n, b)) : 0;
        if (t == 0) {
            count[d] = entries < cap ? entries : cap;
            if (entries > cap) atomicOr(flags, FLAG_CAPACITY);
        }
        // sweep vertices j >= ja, then the other static vertices k >= ka
        for (int64_t q = t; q < m + n && entries > 0; q += CONS_THREADS) {
            int64_t j, k;  // cells that hold the piece from this vertex on
            double p1;
            int64_t place;
            if (q < m) {
                if (q < ja) continue;
                j = q;
                p1 = R.xs(j);
                if (!(p1 < b)) continue;
                k = first_above(xt, n, p1) - 1;
                place = place_before(j, first_not_below(xt, n, p1));
            } else {
                k = q - m;
                if (k < ka || rank[k + 1] == rank[k]) continue;
                p1 = R.xt(k);
                if (!(p1 < b)) continue;
                j = first_above(xs, m, p1) - 1;
                place = place_before(j + 1, k);
            }
            const double p2 = fmin(R.xs(j + 1), R.xt(k + 1));
            // the saved place: inputs in order of their saved index, each
            // input's entries in order of their output's
            const double c1 = fmin(R.xs(j + 1), b);
            const double c0 = fmax(R.xs(j), a);
            const int64_t first = place_before(c0 == R.xs(j) ? j : ja, first_not_below(xt, n, c0));
            const int64_t last = place_before(first_not_below(xs, m, c1), first_not_below(xt, n, c1));
            int64_t at = place;
            if (R.rev_in && R.rev_out) at = entries - 1 - place;
            else if (R.rev_out) at = first + last - 1 - place;
            else if (R.rev_in) at = entries - last + place - first;
            if (at >= cap) continue;
            o_in[at] = R.rev_in ? ~j : j;
            o_out[at] = R.rev_out ? ~k : k;
            o_val[at] = R.weight(p1, p2, j, w_row);
        }
        __syncthreads();
    }
}

// A thread per row: the listed ones (list null: all nd).
__global__ void __launch_bounds__(128)
    conservative_1d_sweeps(const double* __restrict__ xin, int64_t in_stride, int64_t m, const double* __restrict__ xout,
                           int64_t out_stride, int64_t n, int64_t nd, const double* __restrict__ w_in, int64_t w_stride,
                           int64_t cap, int64_t* __restrict__ ind_in, int64_t* __restrict__ ind_out,
                           double* __restrict__ val, int64_t* __restrict__ count, unsigned* flags,
                           const int32_t* __restrict__ list, int64_t n_list) {
    const int64_t total = list ? n_list : nd;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t d = list ? list[q] : q;
        const Row1d R(xin + d * in_stride, xout + d * out_stride, m, n);
        count[d] = sweep_1d(R, w_in ? w_in + d * w_stride : nullptr, cap, ind_in + d * cap, ind_out + d * cap,
                            val + d * cap, flags);
    }
}

__global__ void cell_length_kernel(const double* x, int64_t nd, int64_t n, double* len) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nd * (n - 1);
         k += (int64_t)gridDim.x * blockDim.x) {
        int64_t d = k / (n - 1), i = k % (n - 1);
        len[k] = dsub(x[d * n + i + 1], x[d * n + i]);
    }
}

__global__ void transpose_scale_kernel(const int64_t* __restrict__ ii, const int64_t* __restrict__ oo,
                                       const double* __restrict__ v, int64_t nnz,
                                       const double* __restrict__ vol_in, int64_t n_in,
                                       const double* __restrict__ vol_out, int64_t n_out,
                                       const double* __restrict__ w_in, double* __restrict__ res) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nnz;
         k += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = ii[k] < 0 ? ii[k] + n_in : ii[k];
        int64_t o = oo[k] < 0 ? oo[k] + n_out : oo[k];
        if (i < 0 || i >= n_in || o < 0 || o >= n_out) {
            res[k] = NAN;  // index outside the grids: no volume to scale by
            continue;
        }
        double x = v[k];
        if (w_in) {
            double wi = w_in[i];
            x = ddiv(x, dmul(wi, wi));
        }
        res[k] = ddiv(dmul(x, vol_in[i]), vol_out[o]);
    }
}

}  // namespace

int find_indices_1d(const double* xin, int64_t in_stride, int64_t m, const double* xout,
                    int64_t out_stride, int64_t n, int64_t nd, int method, int64_t fill,
                    int64_t* res, cudaStream_t s) {
    RG_CHECK(method == 0 || method == 1, RG_ERR_ARG, "find_indices: unknown method %d", method);
    if (nd * n <= 0) return RG_OK;
    RG_CHECK(m >= 1, RG_ERR_ARG, "find_indices: empty input grid");
    uint8_t* sorted = nullptr;
    int64_t nrows = in_stride ? nd : 1;
    if (method == 0) {
        RG_TRY(dalloc(&sorted, (size_t)nrows, s));
        row_sorted_kernel<<<grid_for(nrows * 32, 256), 256, 0, s>>>(xin, in_stride, m, nrows, sorted);
    }
    unsigned g = grid_for(nd * n, 256);
    if (g > 65536) g = 65536;
    find_indices_kernel<<<g, 256, 0, s>>>(xin, in_stride, m, xout, out_stride, n, nd, method, fill,
                                          sorted, res);
    dfree(sorted, s);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

int multilinear_1d(const double* xin, int64_t in_stride, int64_t m, const double* xout,
                   const double* xsearch, int64_t out_stride, int64_t n, int64_t nd, const double* w_in,
                   int64_t w_stride,
                   int bounds, int64_t* ind_in, int64_t* ind_out, double* val, int64_t* h_n_outside,
                   cudaStream_t s) {
    RG_CHECK(m >= 2, RG_ERR_ARG, "multilinear: the input grid needs at least 2 vertices");
    RG_CHECK(bounds >= 0 && bounds <= 2, RG_ERR_ARG, "multilinear: unknown bounds %d", bounds);
    int64_t total = 2 * n * nd;
    if (total == 0) return RG_OK;
    RG_CHECK(nd * m < INT32_MAX, RG_ERR_UNSUPPORTED,
             "multilinear: rows x input vertices must stay below 2^31");
    int32_t* bucket = nullptr;
    int64_t* skey = nullptr;
    double* raw_val = nullptr;
    int64_t* bptr = nullptr;
    uint32_t* perm = nullptr;
    unsigned long long* nout = nullptr;
    int st = RG_OK;
    do {
        if ((st = dalloc(&bucket, (size_t)total, s))) break;
        if ((st = dalloc(&skey, (size_t)total, s))) break;
        if ((st = dalloc(&raw_val, (size_t)total, s))) break;
        if ((st = dalloc(&nout, 1, s))) break;
        cudaMemsetAsync(nout, 0, sizeof(unsigned long long), s);
        unsigned g = grid_for(nd * n, 256);
        if (g > 65536) g = 65536;
        multilinear_kernel<<<g, 256, 0, s>>>(xin, in_stride, m, xout, xsearch, out_stride, n, nd, w_in, w_stride,
                                             bounds, bucket, skey, raw_val, nout);
        if (bounds == RG_BOUNDS_RAISE || h_n_outside) {
            unsigned long long h = 0;
            cudaMemcpyAsync(&h, nout, sizeof(h), cudaMemcpyDeviceToHost, s);
            cudaError_t e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) {
                set_error("multilinear: %s", cudaGetErrorString(e));
                st = RG_ERR_CUDA;
                break;
            }
            if (h_n_outside) *h_n_outside = (int64_t)h;
            if (bounds == RG_BOUNDS_RAISE && h) break;
        }
        if ((st = dalloc(&bptr, (size_t)(nd * m) + 1, s))) break;
        if ((st = dalloc(&perm, (size_t)total, s))) break;
        if ((st = bucket_sort(bucket, skey, total, nd * m, bptr, perm, nullptr, s))) break;
        g = grid_for(total, 256);
        if (g > 65536) g = 65536;
        gather_multilinear<<<g, 256, 0, s>>>(perm, bucket, skey, raw_val, total, m, ind_in, ind_out, val);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_error("multilinear: %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
        }
    } while (0);
    dfree(bucket, s);
    dfree(skey, s);
    dfree(raw_val, s);
    dfree(bptr, s);
    dfree(perm, s);
    dfree(nout, s);
    return st;
}

// Whether a thread takes each row (else a block).  A block takes about 20 ns
// and 0.17 ns a vertex of a row, the chip over; a thread 3.3 us a vertex at most,
// for as many rows as run at a time.  Blocks and threads, us: rows of 64 and 48
// vertices, 3,000: 134 and 150, 6,000: 250 and 150, 100,000: 3650 and 550 (one of
// the grids reversed: 610); of 17 and 9, 4,000: 130 and 57; of 513 and 385, 10,000:
// 1610 and 1120, 20,000: 3180 and 1580 (reversed 2770).
static bool rows_by_threads(int64_t nd, int64_t m, int64_t n) {
    return nd * (20 + 0.17 * (m + n)) > 3300.0 * (m + n);
}

int conservative_1d(const double* xin, int64_t in_stride, int64_t m, const double* xout,
                    int64_t out_stride, int64_t n, int64_t nd, const double* w_in, int64_t w_stride,
                    int64_t cap, int64_t* ind_in, int64_t* ind_out, double* val, int64_t* count,
                    cudaStream_t s) {
    RG_CHECK(m >= 2 && n >= 2, RG_ERR_ARG, "conservative 1D: grids need at least 2 vertices");
    if (nd <= 0) return RG_OK;
    RG_CHECK(nd * (m - 1) < INT32_MAX && nd * cap < UINT32_MAX, RG_ERR_UNSUPPORTED,
             "conservative 1D: batch too large");
    const bool threads = rows_by_threads(nd, m, n);
    // uneven rows swept in place: all, where every block has one row at most
    const unsigned blocks = (unsigned)std::min<int64_t>(nd, 152 * 8), few = nd <= blocks ? blocks : 32;
    unsigned* flags = nullptr;  // conditions met, the uneven rows' count, and the list of those past `few`
    int* rank = nullptr;
    int32_t* list = nullptr;
    int st = RG_OK;
    do {
        if ((st = dalloc(&flags, 2 + (threads ? 0 : (size_t)(nd - std::min<int64_t>(nd, few))), s))) break;
        if ((st = zero_async(flags, 2 * sizeof(unsigned), s))) break;
        const auto sweeps = [&](int64_t rows) {
            conservative_1d_sweeps<<<std::min(grid_for(rows, 128), 152u * 16u), 128, 0, s>>>(
                xin, in_stride, m, xout, out_stride, n, nd, w_in, w_stride, cap, ind_in, ind_out, val, count, flags, list, rows);
        };
        unsigned fl[2] = {0, 0};
        const auto read = [&]() {
            small_to_host(fl, flags, sizeof(fl), s);
            const cudaError_t e = cudaStreamSynchronize(s);
            if (e == cudaSuccess) return (int)RG_OK;
            set_error("conservative 1D: %s", cudaGetErrorString(e));
            return (int)RG_ERR_CUDA;
        };
        if (threads) {
            sweeps(nd);
            if ((st = read())) break;
        } else {
            list = (int32_t*)(flags + 2);
            // the ranks of a row's static vertices: shared memory up to 8191 of them
            const size_t shared = n < 8192 ? (size_t)(n + 1) * sizeof(int) : 0;
            if (shared == 0 && (st = dalloc(&rank, (size_t)blocks * (n + 1), s))) break;
            conservative_1d_rows<<<blocks, CONS_THREADS, shared, s>>>(xin, in_stride, m, xout, out_stride, n, nd, w_in,
                                                                      w_stride, cap, ind_in, ind_out, val, count, rank,
                                                                      flags, list, flags + 1, few);
            if ((st = read())) break;
            if (fl[1] > few) {
                sweeps(fl[1] - few);
                if ((st = read())) break;
            }
        }
        if (fl[0] & FLAG_CAPACITY) {
            set_error("conservative 1D: per-row capacity %lld exceeded", (long long)cap);
            st = RG_ERR_ARG;
        }
    } while (0);
    dfree(rank, s);
    dfree(flags, s);
    return st;
}

int cell_length_1d(const double* x, int64_t nd, int64_t n, double* len, cudaStream_t s) {
    if (nd * (n - 1) <= 0) return RG_OK;
    unsigned g = grid_for(nd * (n - 1), 256);
    if (g > 65536) g = 65536;
    cell_length_kernel<<<g, 256, 0, s>>>(x, nd, n, len);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

int transpose_conservative_scale(const int64_t* ii, const int64_t* oo, const double* v, int64_t nnz,
                                 const double* vol_in, int64_t n_in, const double* vol_out,
                                 int64_t n_out, const double* w_in, double* res, cudaStream_t s) {
    if (nnz <= 0) return RG_OK;
    unsigned g = grid_for(nnz, 256);
    if (g > 65536) g = 65536;
    transpose_scale_kernel<<<g, 256, 0, s>>>(ii, oo, v, nnz, vol_in, n_in, vol_out, n_out, w_in, res);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

namespace {

// ndarray_linear_interpolation (regridding/_interp_ndarray.py:166-268): one
// thread per output point; element e of the orthogonal batch reads its
// samples at a + e * a_stride (stride 0: one array for all elements) and its
// indices at x + e * i_stride (likewise).  The cell is floor(x) moved into
// [0, n - 2] (linear extrapolation outside, :208-213), and the point formulas
// keep the upstream operation order with one rounding per operation.  The
// host guarantees n >= 2 on every interpolated axis, so all four reads stay
// inside the array; floor() of a huge or NaN index converts with saturation
// and is then clamped like any other.
__device__ __forceinline__ int64_t interp_cell(double v, int64_t n) {
    int64_t c = (int64_t)floor(v);
    if (c < 0) c = 0;
    else if (c > n - 2) c = n - 2;
    return c;
}

// The per-point part of the upstream formulas: the cell and the weights
// (1D: w00 = 1 - dx, w10 = dx).  When every element shares the points it is
// computed once per point and reused for all the elements a thread visits,
// which halves the FP64 operations per output value (the FP64 pipe, not HBM,
// bounds this kernel on GB300).
struct InterpPoint {
    int64_t i0, j0;
    double w00, w01, w10, w11;
};

__device__ __forceinline__ InterpPoint interp_point(double xv, double yv, int64_t nx, int64_t ny) {
    InterpPoint q;
    q.i0 = interp_cell(xv, nx);
    const double dx = dsub(xv, (double)q.i0);
    if (ny == 0) {
        q.j0 = 0;
        q.w00 = dsub(1.0, dx);
        q.w10 = dx;
        q.w01 = q.w11 = 0.0;
    } else {
        q.j0 = interp_cell(yv, ny);
        const double dy = dsub(yv, (double)q.j0);
        q.w00 = dmul(dsub(1.0, dx), dsub(1.0, dy));
        q.w01 = dmul(dsub(1.0, dx), dy);
        q.w10 = dmul(dx, dsub(1.0, dy));
        q.w11 = dmul(dx, dy);
    }
    return q;
}

// a0 * (1 - dx) + a1 * dx (:217), and (a00 * w00) + (a01 * w01) + (a10 * w10)
// + (a11 * w11) left to right (:268).
__device__ __forceinline__ double interp_eval(const double* __restrict__ s, const InterpPoint& q, int64_t ny) {
    if (ny == 0) return dadd(dmul(s[q.i0], q.w00), dmul(s[q.i0 + 1], q.w10));
    const double* r0 = s + q.i0 * ny + q.j0;
    const double* r1 = r0 + ny;
    return dadd(dadd(dadd(dmul(r0[0], q.w00), dmul(r0[1], q.w01)), dmul(r1[0], q.w10)), dmul(r1[1], q.w11));
}

// Thread = one point p for a run of `run` consecutive elements (grid y);
// reads of each element's samples by neighbouring threads fall on
// neighbouring points, and the output rows are written coalesced.
__global__ void interp_kernel(const double* __restrict__ a, int64_t a_stride, int64_t nx, int64_t ny,
                              const double* __restrict__ x, const double* __restrict__ y, int64_t i_stride,
                              int64_t m, int64_t n_orth, int64_t run, double* __restrict__ out) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < m; p += (int64_t)gridDim.x * blockDim.x) {
        for (int64_t e0 = blockIdx.y * run; e0 < n_orth; e0 += (int64_t)gridDim.y * run) {
            const int64_t e1 = e0 + run < n_orth ? e0 + run : n_orth;
            if (i_stride == 0) {
                const InterpPoint q = interp_point(x[p], ny ? y[p] : 0.0, nx, ny);
                for (int64_t e = e0; e < e1; ++e) out[e * m + p] = interp_eval(a + e * a_stride, q, ny);
            } else {
                for (int64_t e = e0; e < e1; ++e) {
                    const int64_t k = e * i_stride + p;
                    const InterpPoint q = interp_point(x[k], ny ? y[k] : 0.0, nx, ny);
                    out[e * m + p] = interp_eval(a + e * a_stride, q, ny);
                }
            }
        }
    }
}

}  // namespace

}  // namespace rg

extern "C" int rg_interp_linear(const double* d_a, int64_t a_stride, int64_t nx, int64_t ny, const double* d_x,
                                const double* d_y, int64_t i_stride, int64_t m, int64_t n_orth, double* d_out,
                                rg_stream_t stream) {
    rg::NvtxRange nvtx_range("rg_interp_linear");
    using namespace rg;
    RG_CHECK(nx >= 2 && (ny == 0 || ny >= 2) && m >= 0 && n_orth >= 0 && a_stride >= 0 && i_stride >= 0, RG_ERR_ARG,
             "rg_interp_linear: every interpolated axis needs at least 2 samples");
    RG_CHECK(ny == 0 || d_y, RG_ERR_ARG, "rg_interp_linear: 2D interpolation needs y indices");
    if (m == 0 || n_orth == 0) return RG_OK;
    RG_CHECK(d_a && d_x && d_out, RG_ERR_ARG, "rg_interp_linear: NULL argument");
    const int64_t run = i_stride == 0 ? (n_orth < 16 ? n_orth : 16) : 1;
    const int64_t runs = (n_orth + run - 1) / run;
    const unsigned gx = grid_for(m, 256) > (1u << 20) ? (1u << 20) : grid_for(m, 256);
    const unsigned gy = runs > 65535 ? 65535u : (unsigned)runs;
    interp_kernel<<<dim3(gx, gy), 256, 0, (cudaStream_t)stream>>>(d_a, a_stride, nx, ny, d_x, d_y, i_stride, m,
                                                                  n_orth, run, d_out);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

