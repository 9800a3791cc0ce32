// The patch kernel with wide boxes (box_state 2): footprints that exceed the
// 32 x 32 swizzled box, and input rows that are no whole 16-byte chunks.
// Without them those handles gathered from global memory, the exact and
// compensated modes with FP64 sums whose lanes ran rows of unequal length.
// Measured, before and after: 2048^2 -> 1536^2 rotated by 0.45 rad, 64 float32
// slices, compensated 7.17 -> 0.60 ms (HBM 0.36 ms; the kernel is bound by its
// instruction stream) and fast 0.50 -> 0.35 ms (a mean over three rotations);
// 1601^2 -> 1201^2, 32 slices, compensated 2.20 -> 0.33 ms; 777 x 611 -> 583 x
// 458, 32 slices, exact 0.44 -> 0.25 ms (FP64 issue).
#include <algorithm>

#include "common.cuh"
#include "patch.cuh"

namespace rg {

bool encode_stack(const rg_weights_state* W, const void* vin, int64_t stack, int bs, int pitch, int bytes, CUtensorMap* map);
PatchGrid patch_grid(const rg_weights_state* W);
BoxShape box_shape(const rg_weights_state* W);

namespace {

// (box: the handle's, or for a handle of swizzled boxes a wide one of the same
// extent)
template <int PL, int SPS, int NST, int MODE, int LOAD, typename TIN>
int launch_wide(const rg_weights_state* W, BoxShape box, const TIN* vin, void* vout, int64_t stack, cudaStream_t s) {
    constexpr int CT = MODE == MODE_FF ? 6 : CACHED_T;
    const auto kernel = apply_patch_tma<SPS, NST, 0, MODE, CT, LOAD, PL, TIN>;
    const size_t smem = (size_t)NST * SPS * PL * sizeof(TIN);
    static SharedLimit limit;
    if (!allow_shared((const void*)kernel, 200 * 1024, limit)) return RG_ERR_UNSUPPORTED;
    CUtensorMap map = {};
    if (!encode_stack(W, vin, stack, 1, box.pitch, (int)sizeof(TIN), &map)) return RG_ERR_UNSUPPORTED;
    const int64_t patches = W->box_patches;
    // split the stack over gridDim.y only when the patches alone give less
    // than ~4 waves of 4 blocks per SM on 152 SMs
    const int64_t target_blocks = 152 * 4 * 4;
    const int64_t chunks = std::max<int64_t>(1, (target_blocks + patches - 1) / patches);
    int64_t chunk = (stack + chunks - 1) / chunks;
    chunk = (chunk + SPS - 1) / SPS * SPS;
    if ((stack + chunk - 1) / chunk > 65535) chunk = ((stack + 65534) / 65535 + SPS - 1) / SPS * SPS;
    const dim3 grid((unsigned)patches, (unsigned)((stack + chunk - 1) / chunk));
    // bytes of one copy: a slice's box, or the rows of one residue
    const int rows = LOAD == LOAD_RESIDUES ? (W->box_rows + 3) / 4 : W->box_rows;
    const unsigned box_bytes = (unsigned)(rows * box.pitch * sizeof(TIN));
    constexpr bool OUT64 = MODE != MODE_FAST;
    constexpr bool FF = MODE == MODE_FF;
    kernel<<<grid, 32 * PATCH_WARPS, smem, s>>>(
        map, W->row_ptr, W->col, FF ? W->ff_slot : W->box_slot, FF ? W->ff_hi : W->box_val, FF ? W->ff_lo : nullptr,
        W->val32, W->val, OUT64 ? (double*)vout : nullptr, FastDiv((uint32_t)W->in_shape1), patch_grid(W), patches,
        W->box_origin, W->box_rows, SPS * PL, box_bytes, vin, W->n_in,
        OUT64 ? nullptr : (float*)vout, W->n_out, stack, chunk, W->dflags,
        FF ? W->ff_perm : (OUT64 ? W->box_perm : nullptr), box, W->box_extent);
    RG_CUDA(cudaGetLastError());
    return RG_OK;
}

// Slices per stage: a stage computes all its slices, also those past the end
// of the stack, so one or two slices take stages of two; the largest boxes
// (from 9 KB a slice) too, to keep three blocks on an SM.
constexpr int FOUR_SLICES = 2304 * 4;  // bytes of a slice's plane, at most
template <int PL, int MODE, int LOAD, typename TIN>
int launch_plane(const rg_weights_state* W, BoxShape box, const TIN* vin, void* vout, int64_t stack, cudaStream_t s) {
    if constexpr (PL * sizeof(TIN) <= FOUR_SLICES)
        if (stack > 2) return launch_wide<PL, 4, 2, MODE, LOAD>(W, box, vin, vout, stack, s);
    return launch_wide<PL, 2, 2, MODE, LOAD>(W, box, vin, vout, stack, s);
}

// A slice's plane in a stage, the smallest of a few sizes that holds the box
// (a constant, so that a gather's slices differ by constant offsets).
int box_cells(const rg_weights_state* W, BoxShape box) { return box.residues ? 4 * box.residues : W->box_rows * box.pitch; }
int plane_cells(int cells) { return cells <= 1024 ? 1024 : cells <= 1536 ? 1536 : cells <= 2304 ? 2304 : 3584; }

template <int MODE, int LOAD, typename TIN>
int launch_mode(const rg_weights_state* W, BoxShape box, const TIN* vin, void* vout, int64_t stack, cudaStream_t s) {
    switch (plane_cells(box_cells(W, box))) {
        case 1024: return launch_plane<1024, MODE, LOAD>(W, box, vin, vout, stack, s);
        case 1536: return launch_plane<1536, MODE, LOAD>(W, box, vin, vout, stack, s);
        case 2304: return launch_plane<2304, MODE, LOAD>(W, box, vin, vout, stack, s);
        default: return launch_plane<3584, MODE, LOAD>(W, box, vin, vout, stack, s);
    }
}

// The box a float64 stack takes with a handle of swizzled ones.
BoxShape narrow_box(const rg_weights_state* W) { return BoxShape{W->in_shape1 >= 36 ? 36 : 32, 0}; }

template <int MODE, typename TIN>
int launch_load(const rg_weights_state* W, int load, const TIN* vin, void* vout, int64_t stack, cudaStream_t s) {
    if (load == LOAD_WIDE) return launch_mode<MODE, LOAD_WIDE>(W, box_shape(W), vin, vout, stack, s);
    if constexpr (MODE != MODE_FAST) return launch_mode<MODE, LOAD_RESIDUES>(W, box_shape(W), vin, vout, stack, s);
    return RG_ERR_UNSUPPORTED;
}

}  // namespace

int apply_wide(const rg_weights_state* W, int mode, int load, const float* vin, void* vout, int64_t stack, cudaStream_t s) {
    switch (mode) {
        case MODE_FAST: return launch_load<MODE_FAST>(W, load, vin, vout, stack, s);
        case MODE_EXACT: return launch_load<MODE_EXACT>(W, load, vin, vout, stack, s);
        default: return launch_load<MODE_FF>(W, load, vin, vout, stack, s);
    }
}

// The exact apply of a float64 stack (box_load, box_perm_for first): as the
// float32 one, in wide boxes also where that takes swizzled ones.
int apply_wide_f64(const rg_weights_state* W, int load, const double* vin, double* vout, int64_t stack, cudaStream_t s) {
    if (load != LOAD_SWIZZLED) return launch_load<MODE_EXACT>(W, load, vin, vout, stack, s);
    return launch_mode<MODE_EXACT, LOAD_WIDE>(W, narrow_box(W), vin, vout, stack, s);
}

// Whether an exact call over cells of `bytes` stages its boxes; gathers from
// global memory give the same bits.  A stage computes all its slices, 2 or 4
// (launch_plane), and a gather none too many, so it hangs on the share that the
// stack fills.  Gathered and staged, us, at 2, 4, 8 and 16 slices (one and two
// float32 slices):
//   float32, wide boxes, 2048^2 -> 1536^2 rotated by 0.45: 216, 427, 850, 1691
//     and 118, 218, 417, 817 (one: 111 and 118);
//     -> 819^2 at 0.1: 167, 326, 645, 1282 and 118, 187, 323, 592 (one: 88, 116);
//   float32, row residues, 777 x 611 -> 583 x 458 at 0.45: 31, 60, 115, 226 and
//     36, 44, 75, 131;
//   float64, boxes of 32 columns, 1024^2 -> 768^2 at 0.1: 46, 88, 172, 337 and
//     44, 66, 120, 221;
//   float64, wide ones of up to 1536 cells, 2048^2 -> 1536^2 at 0.45: 152, 294,
//     579, 1150 and 145, 272, 525, 1039;
//   float64, row residues, 777 x 611 at 0.45: 24, 42, 79, 156 and 40, 44, 72, 126;
//   float64, above 1536 cells, 1000 x 700 -> 500 x 350 at 4, 8, 16: 48, 89, 171
//     and 55, 95, 150.
bool exact_staged(const rg_weights_state* W, int load, int bytes, int64_t stack) {
    if (bytes == 4 && load == LOAD_SWIZZLED) return true;
    const int cells = box_cells(W, load == LOAD_SWIZZLED ? narrow_box(W) : box_shape(W));
    const int per = plane_cells(cells) * bytes <= FOUR_SLICES && stack > 2 ? 4 : 2;
    const int64_t computed = (stack + per - 1) / per * per;
    const bool residues = load == LOAD_RESIDUES;
    if (bytes == 4) return 2 * computed <= 3 * stack && (!residues || stack >= 3);
    if (load == LOAD_SWIZZLED) return 3 * computed <= 4 * stack;
    return 100 * computed <= 108 * stack && stack >= (cells > 1536 ? 16 : residues ? 8 : 2);
}

}  // namespace rg
