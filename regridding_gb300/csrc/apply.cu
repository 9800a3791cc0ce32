// Apply of device-resident weights to a stack of arrays:
//   values_output[d, o] = sum_k w[o, k] * values_input[d, col[o, k]]
// (regridding/_regrid/_regrid_from_weights.py:165-182).
//
// The matrix is stored by output row, so every output element is produced by
// exactly one thread with no atomics.  A block covers a 2D tile of output
// cells (8 x 32 when the output grid shape is known, so the input footprint of
// the block is compact and its gathers reuse L1/L2 lines) and a chunk of the
// stack; each thread keeps its row's first entries in registers and walks the
// stack chunk, so the weights are read once per chunk instead of once per
// array.
#include "common.cuh"
#include "patch.cuh"

namespace rg {
namespace {

constexpr int APPLY_BLOCK = 256;
constexpr int CACHED = 8;  // row entries held in registers

template <typename T>
__device__ __forceinline__ T ldg_cast(const T* p) { return __ldg(p); }

struct Tile {
    int64_t n0, n1;  // output shape used for tiling (n0 = 1 for 1D tiling)
    int64_t tiles1;  // tiles along axis 1
    int t0, t1;      // tile extent
};

__device__ __forceinline__ int64_t tile_row(const Tile& T, int64_t tile, int tid) {
    int64_t ti = tile / T.tiles1, tj = tile % T.tiles1;
    int64_t i = ti * T.t0 + tid / T.t1;
    int64_t j = tj * T.t1 + tid % T.t1;
    if (i >= T.n0 || j >= T.n1) return -1;
    return i * T.n1 + j;
}

// MODE 0: exact double (mul then add, stored order), float64 output
// MODE 1: exact double update rounded to float32 after every entry (numpy's
//         in-place float32 output)
// MODE 2: fast, accumulate in the output type with FMA
// MODE 3: compensated (float32 input, float64 output): rows of up to FF_ROW_MAX
//         entries by the float-float sums of the patch kernel, two slices at a
//         time, for footprints too large for its boxes (777 x 611 -> 311 x 244
//         rotated by 0.45, 8 slices: 91 us as MODE 0, 44 so); longer ones as
//         MODE 0
template <typename Tin, typename Tout, int MODE, typename Tw>
__global__ void __launch_bounds__(APPLY_BLOCK)
    apply_kernel(const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                 const Tw* __restrict__ val, Tile T, const Tin* __restrict__ vin, int64_t n_in,
                 Tout* __restrict__ vout, int64_t n_out, int64_t stack, int64_t chunk) {
    int64_t o = tile_row(T, blockIdx.x, threadIdx.x);
    if (o < 0) return;
    int64_t d0 = (int64_t)blockIdx.y * chunk;
    int64_t d1 = d0 + chunk < stack ? d0 + chunk : stack;
    int64_t s = row_ptr[o], e = row_ptr[o + 1];
    int nk = (int)(e - s);
    int32_t c[CACHED];
    Tw w[CACHED];
#pragma unroll
    for (int k = 0; k < CACHED; k++) {
        c[k] = k < nk ? col[s + k] : 0;
        w[k] = k < nk ? val[s + k] : (Tw)0;
    }
    if constexpr (MODE == 3) {
        if (nk <= FF_ROW_MAX) {
            float hi[CACHED], lo[CACHED];
#pragma unroll
            for (int k = 0; k < CACHED; k++) {
                hi[k] = (float)w[k];
                lo[k] = __double2float_rn(__dsub_rn(w[k], (double)hi[k]));
            }
            for (int64_t d = d0; d < d1; d += 2) {
                const Tin* a = vin + d * n_in;
                const Tin* b = d + 1 < d1 ? a + n_in : a;
                uint64_t h2 = 0ull, l2 = 0ull;
                auto step = [&](int32_t cell, float wh, float wl) {
                    ff_step2(h2, l2, f2_pack(wh, wh), f2_pack(-wh, -wh), f2_pack(wl, wl),
                             f2_pack(ldg_cast(a + cell), ldg_cast(b + cell)));
                };
#pragma unroll
                for (int k = 0; k < CACHED; k++)
                    if (k < nk) step(c[k], hi[k], lo[k]);
                for (int64_t k = s + CACHED; k < e; k++) {
                    const float wh = (float)val[k];
                    step(col[k], wh, __double2float_rn(__dsub_rn(val[k], (double)wh)));
                }
                const float2 h = f2_unpack(h2), l = f2_unpack(l2);
                auto store = [&](int64_t dd, const Tin* x, float hv, float lv) {
                    double r = 0.0;
                    if (finite_bits(hv) && finite_bits(lv)) {
                        r = __dadd_rn(widen(hv), widen(lv));
                    } else {  // as the patch kernel: this output and slice in float64, stored order
                        for (int64_t k = s; k < e; k++)
                            r = __dadd_rn(r, __dmul_rn((double)val[k], (double)ldg_cast(x + col[k])));
                    }
                    vout[dd * n_out + o] = (Tout)r;
                };
                store(d, a, h.x, l.x);
                if (d + 1 < d1) store(d + 1, b, h.y, l.y);
            }
            return;
        }
    }
    for (int64_t d = d0; d < d1; d++) {
        const Tin* a = vin + d * n_in;
        if (MODE == 0 || MODE == 3) {
            double acc = 0.0;
#pragma unroll
            for (int k = 0; k < CACHED; k++)
                if (k < nk) acc = __dadd_rn(acc, __dmul_rn((double)w[k], (double)ldg_cast(a + c[k])));
            for (int64_t k = s + CACHED; k < e; k++)
                acc = __dadd_rn(acc, __dmul_rn((double)val[k], (double)ldg_cast(a + col[k])));
            vout[d * n_out + o] = (Tout)acc;
        } else if (MODE == 1) {
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k < CACHED; k++)
                if (k < nk)
                    acc = (float)__dadd_rn((double)acc, __dmul_rn((double)w[k], (double)ldg_cast(a + c[k])));
            for (int64_t k = s + CACHED; k < e; k++)
                acc = (float)__dadd_rn((double)acc, __dmul_rn((double)val[k], (double)ldg_cast(a + col[k])));
            vout[d * n_out + o] = (Tout)acc;
        } else {
            Tout acc = (Tout)0;
#pragma unroll
            for (int k = 0; k < CACHED; k++)
                if (k < nk) acc = fma((Tout)w[k], (Tout)ldg_cast(a + c[k]), acc);
            for (int64_t k = s + CACHED; k < e; k++) acc = fma((Tout)val[k], (Tout)ldg_cast(a + col[k]), acc);
            vout[d * n_out + o] = acc;
        }
    }
}

__global__ void to_f32(const double* a, float* b, int64_t n) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x)
        b[k] = (float)a[k];
}

template <typename Tin, typename Tout, int MODE, typename Tw>
int launch(const int64_t* row_ptr, const int32_t* col, const Tw* val, int64_t n_rows,
           int64_t shape0, int64_t shape1, const void* vin, int64_t n_in, void* vout, int64_t stack,
           cudaStream_t s) {
    Tile T;
    if (shape0 > 0 && shape1 > 0 && shape0 * shape1 == n_rows && shape1 >= 32) {
        T.n0 = shape0;
        T.n1 = shape1;
        T.t0 = 8;
        T.t1 = 32;
    } else {
        T.n0 = 1;
        T.n1 = n_rows;
        T.t0 = 1;
        T.t1 = APPLY_BLOCK;
    }
    T.tiles1 = (T.n1 + T.t1 - 1) / T.t1;
    int64_t tiles = ((T.n0 + T.t0 - 1) / T.t0) * T.tiles1;
    // stack chunk: enough blocks to fill the GPU, at most 65535 along y
    int64_t chunk = 16;
    if (tiles >= 4 * 152 * 8) chunk = 64;
    if ((stack + chunk - 1) / chunk > 65535) chunk = (stack + 65534) / 65535;
    int64_t chunks = (stack + chunk - 1) / chunk;
    RG_CHECK(tiles < 0x7fffffff, RG_ERR_UNSUPPORTED, "apply: too many output cells");
    dim3 grid((unsigned)tiles, (unsigned)chunks);
    apply_kernel<Tin, Tout, MODE, Tw><<<grid, APPLY_BLOCK, 0, s>>>(
        row_ptr, col, val, T, (const Tin*)vin, n_in, (Tout*)vout, n_rows, stack, chunk);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

int apply_csr(const int64_t* row_ptr, const int32_t* col, const double* val, const float* val32,
              int64_t nnz, int64_t n_rows, int64_t n_cols, int64_t shape0, int64_t shape1,
              const void* vin, int dtype_in, void* vout, int dtype_out, int64_t stack, int acc,
              cudaStream_t s) {
    RG_CHECK(dtype_in == RG_F32 || dtype_in == RG_F64, RG_ERR_ARG, "apply: bad input dtype");
    RG_CHECK(dtype_out == RG_F32 || dtype_out == RG_F64, RG_ERR_ARG, "apply: bad output dtype");
    RG_CHECK(acc == RG_ACC_EXACT || acc == RG_ACC_FAST || acc == RG_ACC_COMPENSATED, RG_ERR_ARG,
             "apply: bad accumulation mode");
    if (stack <= 0 || n_rows <= 0) return RG_OK;
    if (acc == RG_ACC_COMPENSATED && dtype_in == RG_F32 && dtype_out == RG_F64)
        return launch<float, double, 3, double>(row_ptr, col, val, n_rows, shape0, shape1, vin, n_cols, vout, stack,
                                                s);
    if (acc != RG_ACC_FAST) {
        if (dtype_out == RG_F64) {
            if (dtype_in == RG_F32)
                return launch<float, double, 0, double>(row_ptr, col, val, n_rows, shape0, shape1, vin, n_cols,
                                                        vout, stack, s);
            return launch<double, double, 0, double>(row_ptr, col, val, n_rows, shape0, shape1, vin, n_cols,
                                                     vout, stack, s);
        }
        if (dtype_in == RG_F32)
            return launch<float, float, 1, double>(row_ptr, col, val, n_rows, shape0, shape1, vin, n_cols, vout,
                                                   stack, s);
        return launch<double, float, 1, double>(row_ptr, col, val, n_rows, shape0, shape1, vin, n_cols, vout,
                                                stack, s);
    }
    if (dtype_out == RG_F64) {
        if (dtype_in == RG_F32)
            return launch<float, double, 2, double>(row_ptr, col, val, n_rows, shape0, shape1, vin, n_cols, vout,
                                                    stack, s);
        return launch<double, double, 2, double>(row_ptr, col, val, n_rows, shape0, shape1, vin, n_cols, vout,
                                                 stack, s);
    }
    // float32 output, fast: the weights rounded to float once (made by the caller)
    if (dtype_in == RG_F32)
        return launch<float, float, 2, float>(row_ptr, col, val32, n_rows, shape0, shape1, vin, n_cols, vout,
                                              stack, s);
    return launch<double, float, 2, float>(row_ptr, col, val32, n_rows, shape0, shape1, vin, n_cols, vout,
                                           stack, s);
}

}  // namespace

int tiled_lists_for(rg_weights_s* W, const float* vin, cudaStream_t s, int* g, bool* made);
int apply_tiled(const rg_weights_state* W, int g, const float* vin, float* vout, int64_t stack, cudaStream_t s);
bool shapes_usable(const rg_weights_state* W, int64_t stack);
bool box_usable(const rg_weights_state* W, int64_t stack);
int box_load(const rg_weights_state* W, const void* vin, int64_t stack);
bool exact_staged(const rg_weights_state* W, int load, int bytes, int64_t stack);
int apply_wide_f64(const rg_weights_state* W, int load, const double* vin, double* vout, int64_t stack, cudaStream_t s);
int box_order_for(rg_weights_s* W, cudaStream_t s, bool* made);
int box_lists_for(rg_weights_s* W, cudaStream_t s, bool* made);
int box_perm_for(rg_weights_s* W, cudaStream_t s, bool* made);
int ff_lists_for(rg_weights_s* W, cudaStream_t s, bool* made);
int apply_box(const rg_weights_state* W, const float* vin, float* vout, int64_t stack, cudaStream_t s);
int apply_box_exact(const rg_weights_state* W, const float* vin, double* vout, int64_t stack, cudaStream_t s);
int apply_box_ff(const rg_weights_state* W, const float* vin, double* vout, int64_t stack, cudaStream_t s);
int tune_box_fast(rg_weights_s* W, const float* vin, float* vout, int64_t stack, cudaStream_t s);
int tune_box_ff(rg_weights_s* W, const float* vin, double* vout, int64_t stack, cudaStream_t s);
int rows_usable(rg_weights_s* W, const float* vin, int64_t stack, cudaStream_t s, bool* made, bool* ok);
int apply_rows_launch(const rg_weights_state* W, const float* vin, float* vout, int64_t stack, cudaStream_t s);
int ensure_transposed(rg_weights_s* W, cudaStream_t s);

// Whether compensated calls sum float pairs (else they compute as exact).
bool float_pairs(const rg_weights_state* W) {
    return W->box_state == 1 || W->box_long * FF_LONG_SHARE <= W->n_out;
}

// Whether an exact (or compensated) call over a float32 stack finds all that
// box_lists_for and its like would make.
bool lists_ready(const rg_weights_state* W, bool ff, int64_t stack) {
    if (W->box_state <= 0) return W->box_state < 0;
    if (!ff || !float_pairs(W)) return W->box_perm != nullptr;
    return W->ff_slot && (W->box_state == 2 || W->box_cfg_ff[stack_class(stack)] != -1);
}

// Every apply goes through here.  The per-handle state an apply needs beyond
// the CSR (the transposed CSR, the float32 copy of the weights, the warp-tile
// lists) is made on first use under the handle's mutex and finished (the
// stream synchronised) before the lock is released, so calls from other
// threads and streams only ever see complete state.  The launches read a copy
// of it taken under the lock.
int apply_weights(rg_weights_s* W, bool transposed, const void* vin, int dtype_in, void* vout,
                  int dtype_out, int64_t stack, int acc, cudaStream_t s) {
    RG_CHECK(dtype_in == RG_F32 || dtype_in == RG_F64, RG_ERR_ARG, "apply: bad input dtype");
    RG_CHECK(dtype_out == RG_F32 || dtype_out == RG_F64, RG_ERR_ARG, "apply: bad output dtype");
    RG_CHECK(acc == RG_ACC_EXACT || acc == RG_ACC_FAST || acc == RG_ACC_COMPENSATED, RG_ERR_ARG,
             "apply: bad accumulation mode");
    if (stack <= 0) return RG_OK;
    // the bandwidth path: float32 in and out, input staged in shared memory (by
    // tensor-map copies when the input grid shape allows, else by the warps)
    const bool tiled = !transposed && acc == RG_ACC_FAST && dtype_in == RG_F32 && dtype_out == RG_F32 &&
                       W->n_out > 0 && W->nnz > 0;
    // the exact float64 apply of a float32 stack stages input boxes too
    const bool exact_box = !transposed && acc == RG_ACC_EXACT && dtype_in == RG_F32 && dtype_out == RG_F64 &&
                           W->n_out > 0 && W->nnz > 0;
    // and that of a float64 stack, from a handle's second such call on: the
    // lists cost about as much as the second and third calls save, and gathers
    // from global memory, which a first call takes, give the same bits
    bool exact64 = !transposed && acc != RG_ACC_FAST && dtype_in == RG_F64 && dtype_out == RG_F64 && W->n_out > 0 &&
                   W->nnz > 0 && stack >= 2;
    // the compensated apply: float32 stack, float64 output, float-float sums
    const bool ff_box = !transposed && acc == RG_ACC_COMPENSATED && dtype_in == RG_F32 && dtype_out == RG_F64 &&
                        W->n_out > 0 && W->nnz > 0;
    // (the patch lists keep a float32 copy of the weights in gather order)
    const bool need32 = ((acc == RG_ACC_FAST && dtype_out == RG_F32) || exact_box || ff_box) && W->nnz > 0;
    int g = 0, load64 = -1;
    bool use_box = false, use_rows = false, use_box_exact = false, use_box_ff = false, ff_direct = false;
    rg_weights_state now;
    {
        std::lock_guard<std::mutex> lock(W->mu);
        bool made = false;
        if (exact64 && !W->box_perm) {
            // (the lists are read back by the host: not while a graph is captured)
            cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
            if (W->exact64_calls++ > 0) RG_CUDA(cudaStreamIsCapturing(s, &capture));
            else exact64 = false;
            exact64 = exact64 && capture == cudaStreamCaptureStatusNone;
        }
        if (transposed && W->t_row_ptr == nullptr) {
            RG_TRY(ensure_transposed(W, s));
            made = true;
        }
        float** v32 = transposed ? &W->t_val32 : &W->val32;
        if (need32 && *v32 == nullptr) {
            RG_TRY(dalloc(v32, (size_t)W->nnz, s));
            to_f32<<<grid_for(W->nnz, 256) > 8192 ? 8192 : grid_for(W->nnz, 256), 256, 0, s>>>(
                transposed ? W->t_val : W->val, *v32, W->nnz);
            made = true;
        }
        if ((tiled || exact_box || ff_box) && W->in_shape1 % 4 == 0 && ((uintptr_t)vin & 15) == 0 && shapes_usable(W, stack))
            W->in_fixed = true;
        // the lists of a call are read back by the host: while a graph is captured
        // float32 stacks with float64 sums gather where they are not there yet
        bool boxes = box_usable(W, stack);
        if ((exact_box || ff_box) && boxes && !lists_ready(W, ff_box, stack)) {
            cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
            RG_CUDA(cudaStreamIsCapturing(s, &capture));
            boxes = capture == cudaStreamCaptureStatusNone;
        }
        int load = -1;  // how the patch kernel fills its stages, -1: it does not take the call
        if (((tiled && W->in_shape1 % 4 == 0) || exact_box || exact64 || ff_box) && boxes) {
            RG_TRY(box_lists_for(W, s, &made));
            load = box_load(W, (const float*)vin, stack);
        }
        // (rows that are no whole 16-byte chunks: the row residues' copies cost
        // the fast mode more than its gathers; 1601^2 -> 1201^2, 32 slices 243 us
        // against 189 us of the warp-staged kernel, where the compensated mode
        // goes from 2200 us of FP64 gathers to 330 us)
        if (tiled && load >= 0 && load != LOAD_RESIDUES) {
            use_box = true;
            RG_TRY(box_order_for(W, s, &made));
            if (load == LOAD_SWIZZLED && W->box_cfg[stack_class(stack)] == -1) {
                if (made) RG_CUDA(cudaStreamSynchronize(s));
                made = false;
                RG_TRY(tune_box_fast(W, (const float*)vin, (float*)vout, stack, s));
            }
            use_box = load != LOAD_SWIZZLED || W->box_cfg[stack_class(stack)] >= 0;
        }
        exact64 = exact64 && load >= 0 && exact_staged(W, load, 8, stack);
        load64 = load;
        if (exact64) RG_TRY(box_perm_for(W, s, &made));
        // compensated calls with too many rows too long for float-float sums, those
        // without shapes and those off a 16-byte boundary of the swizzled box
        // compute as exact; footprints too large for any box gather
        ff_direct = ff_box && W->box_state == -1;
        const bool ff_rows = float_pairs(W);
        if ((exact_box || (ff_box && !ff_rows)) && load >= 0 && exact_staged(W, load, 4, stack)) {
            use_box_exact = true;
            RG_TRY(box_perm_for(W, s, &made));
        }
        if (ff_box && ff_rows && load >= 0) {
            use_box_ff = true;
            RG_TRY(ff_lists_for(W, s, &made));
            if (load == LOAD_SWIZZLED && W->box_cfg_ff[stack_class(stack)] == -1) {
                if (made) RG_CUDA(cudaStreamSynchronize(s));
                made = false;
                RG_TRY(tune_box_ff(W, (const float*)vin, (double*)vout, stack, s));
            }
            use_box_ff = load != LOAD_SWIZZLED || W->box_cfg_ff[stack_class(stack)] >= 0;
        }
        if (tiled && !use_box)
            RG_TRY(rows_usable(W, (const float*)vin, stack, s, &made, &use_rows));
        if (tiled && !use_box && !use_rows) RG_TRY(tiled_lists_for(W, (const float*)vin, s, &g, &made));
        if (made) RG_CUDA(cudaStreamSynchronize(s));
        now = *W;
    }
    if (exact64) {
        const int st = apply_wide_f64(&now, load64, (const double*)vin, (double*)vout, stack, s);
        if (st != RG_ERR_UNSUPPORTED) return st;
    }
    if (use_rows) {
        const int st = apply_rows_launch(&now, (const float*)vin, (float*)vout, stack, s);
        if (st != RG_ERR_UNSUPPORTED) return st;
    }
    if (use_box_exact) {
        const int st = apply_box_exact(&now, (const float*)vin, (double*)vout, stack, s);
        if (st != RG_ERR_UNSUPPORTED) return st;
    }
    if (use_box_ff) {
        const int st = apply_box_ff(&now, (const float*)vin, (double*)vout, stack, s);
        if (st != RG_ERR_UNSUPPORTED) return st;
    }
    if (use_box) {
        const int st = apply_box(&now, (const float*)vin, (float*)vout, stack, s);
        if (st != RG_ERR_UNSUPPORTED) return st;
    }
    if (use_rows || use_box) {
        // the tuned configuration does not take this call (fewer slices than
        // a stage), or the device not the kernel's shared memory: the
        // warp-staged kernel does, with its own lists
        std::lock_guard<std::mutex> lock(W->mu);
        bool made = false;
        RG_TRY(tiled_lists_for(W, (const float*)vin, s, &g, &made));
        if (made) RG_CUDA(cudaStreamSynchronize(s));
        now = *W;
    }
    if (tiled) return apply_tiled(&now, g, (const float*)vin, (float*)vout, stack, s);
    if (!transposed)
        return apply_csr(now.row_ptr, now.col, now.val, now.val32, now.nnz, now.n_out, now.n_in, now.out_shape0,
                         now.out_shape1, vin, dtype_in, vout, dtype_out, stack,
                         acc == RG_ACC_COMPENSATED && !ff_direct ? RG_ACC_EXACT : acc, s);
    // (a compensated call is defined for the matrix itself; its transpose computes as exact)
    return apply_csr(now.t_row_ptr, now.t_col, now.t_val, now.t_val32, now.nnz, now.n_in, now.n_out, 0, 0, vin,
                     dtype_in, vout, dtype_out, stack,
                     acc == RG_ACC_COMPENSATED ? RG_ACC_EXACT : acc, s);
}

}  // namespace rg

// ---------------------------------------------------------------------------
// apply with the stack in host memory: the stack is cut into chunks that are
// copied in, applied and copied out on three streams, so the two copy
// directions and the kernels overlap (double-buffered staging in HBM).
// ---------------------------------------------------------------------------
namespace rg {

int apply_host(rg_weights_s* W, const void* h_vin, int dtype_in, void* h_vout, int dtype_out,
               int64_t stack, int acc, int64_t chunk, cudaStream_t s) {
    RG_CHECK(dtype_in == RG_F32 || dtype_in == RG_F64, RG_ERR_ARG, "apply_host: bad input dtype");
    RG_CHECK(dtype_out == RG_F32 || dtype_out == RG_F64, RG_ERR_ARG, "apply_host: bad output dtype");
    if (stack <= 0) return RG_OK;
    const size_t bin = (dtype_in == RG_F32 ? 4 : 8) * (size_t)W->n_in;
    const size_t bout = (dtype_out == RG_F32 ? 4 : 8) * (size_t)W->n_out;
    if (chunk <= 0) {
        // about 128 MB of input per chunk, at least one slice
        chunk = (int64_t)((128u << 20) / (bin ? bin : 1));
        if (chunk < 1) chunk = 1;
    }
    if (chunk > stack) chunk = stack;
    const int64_t nchunks = (stack + chunk - 1) / chunk;

    cudaStream_t sin = nullptr, sout = nullptr;
    cudaEvent_t ev[2 * 3] = {};
    char* dbuf[4] = {};
    int st = RG_OK;
    do {
        if (cudaStreamCreateWithFlags(&sin, cudaStreamNonBlocking) != cudaSuccess ||
            cudaStreamCreateWithFlags(&sout, cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            set_error("apply_host: stream creation failed");
            st = RG_ERR_CUDA;
            break;
        }
        for (int k = 0; k < 6; k++)
            if (cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                set_error("apply_host: event creation failed");
                st = RG_ERR_CUDA;
            }
        if (st) break;
        for (int b = 0; b < 2; b++) {
            if ((st = dalloc(&dbuf[b], bin * chunk, s))) break;
            if ((st = dalloc(&dbuf[2 + b], bout * chunk, s))) break;
        }
        if (st) break;
        // ev[0..1]: input buffer b consumed by the kernel; ev[2..3]: output
        // buffer b copied out; ev[4]: input copy of the current chunk landed;
        // ev[5]: kernel of the current chunk done
        cudaEventRecord(ev[0], s);
        cudaEventRecord(ev[1], s);
        cudaEventRecord(ev[2], s);
        cudaEventRecord(ev[3], s);
        for (int64_t c = 0; c < nchunks && st == RG_OK; c++) {
            int b = (int)(c & 1);
            int64_t d0 = c * chunk, nd = stack - d0 < chunk ? stack - d0 : chunk;
            cudaStreamWaitEvent(sin, ev[b], 0);
            cudaMemcpyAsync(dbuf[b], (const char*)h_vin + d0 * bin, bin * nd, cudaMemcpyHostToDevice, sin);
            cudaEventRecord(ev[4], sin);
            cudaStreamWaitEvent(s, ev[4], 0);
            cudaStreamWaitEvent(s, ev[2 + b], 0);
            st = apply_weights(W, false, dbuf[b], dtype_in, dbuf[2 + b], dtype_out, nd, acc, s);
            cudaEventRecord(ev[b], s);
            cudaEventRecord(ev[5], s);
            cudaStreamWaitEvent(sout, ev[5], 0);
            cudaMemcpyAsync((char*)h_vout + d0 * bout, dbuf[2 + b], bout * nd, cudaMemcpyDeviceToHost, sout);
            cudaEventRecord(ev[2 + b], sout);
        }
        // the caller's stream completes after the last copy out
        cudaStreamWaitEvent(s, ev[2], 0);
        cudaStreamWaitEvent(s, ev[3], 0);
        cudaError_t e = cudaGetLastError();
        if (st == RG_OK && e != cudaSuccess) {
            set_error("apply_host: %s", cudaGetErrorString(e));
            st = RG_ERR_CUDA;
        }
    } while (0);
    for (int b = 0; b < 4; b++) dfree(dbuf[b], s);
    for (int k = 0; k < 6; k++)
        if (ev[k]) cudaEventDestroy(ev[k]);
    if (sin) cudaStreamDestroy(sin);
    if (sout) cudaStreamDestroy(sout);
    return st;
}

}  // namespace rg
