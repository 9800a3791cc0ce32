// The patch kernel of the staged applies (apply_patch_tma) and what its
// preparation shares with it; included by the files that launch it.
#pragma once

#include <cuda.h>  // CUtensorMap

#include "common.cuh"

namespace rg {
namespace {

constexpr int CACHED_T = 8;     // row entries kept in registers across slices
constexpr int FF_EXTRA = 3;     // compensated mode: further row entries kept in shared memory
constexpr int ROW_EXTRA = 2;    // fast and exact modes: further row entries kept in shared memory

// Direct gathers for one lane's row (tiles whose list does not fit).
__device__ __forceinline__ void apply_direct(const int64_t s, const int64_t e, const int32_t* __restrict__ col,
                                             const float* __restrict__ val, const float* __restrict__ vin,
                                             int64_t n_in, float* out, int64_t n_out, int64_t d0, int64_t d1) {
    for (int64_t d = d0; d < d1; d++) {
        const float* a = vin + d * n_in;
        float acc = 0.f;
        for (int64_t k = s; k < e; k++) acc = fmaf(val[k], __ldg(a + col[k]), acc);
        out[d * n_out] = acc;
    }
}

// ---------------------------------------------------------------------------
// TMA variant.  A block of 8 warps owns a 16 x 16 patch of output cells
// (4 x 2 warp tiles of 4 x 8).  The input footprint of every patch lies in a
// box of box_rows x 32 input cells (the same box size for all patches, the
// origin per patch, its column a multiple of 4 so that a copy starts on a
// 16-byte boundary).  A ring of NST stages, each holding SPS slices of the
// patch's box, is filled by one 3D tensor copy per stage (columns x rows x
// slices) issued by thread 0 and completed by the stage's "full" mbarrier
// transaction count; every warp arrives on the stage's "empty" mbarrier when
// it has read the stage, and thread 0 waits for all 8 before refilling it.
// The copies run on the TMA unit, so the load/store pipe only carries the
// gathers of the reduction (one 32-bit shared load per entry and slice).
// Box rows are 128 bytes and written with the 128-byte swizzle (16-byte
// chunk c of row r lands at chunk c ^ (r & 7) of that row), which spreads
// the gathers of vertically neighbouring cells over different banks; the
// entries' slots carry the swizzle.  Waits are bounded: a copy that does not
// land sets FLAG_TIMEOUT and the block leaves after a bounded drain.
// ---------------------------------------------------------------------------

constexpr int PATCH_WARPS = 8; // warp tiles of a patch of 256 output cells
constexpr int PBOX_C = 32;     // box columns: one 128-byte swizzle span
constexpr int PBOX_MAX_R = 32; // box rows at most
constexpr int PLANE = PBOX_MAX_R * PBOX_C;  // floats of one slice's plane in a stage (4 KB)

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// try_wait with a suspend-time hint (ns): the thread sleeps instead of spinning
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}
// bounded wait: gives up after 2^16 polls (each suspends at most ~20 us)
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity) {
    for (int it = 0; it < (1 << 16); it++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

struct PatchGrid {
    int64_t n0, n1;     // output cells
    int64_t patches1;   // patches along axis 1
    int cb;             // a patch is (256 >> cb) x (1 << cb) output cells
};

__device__ __forceinline__ int64_t patch_cell(const PatchGrid& P, int64_t p, int r, int c) {
    const int64_t pi = p / P.patches1, pj = p - pi * P.patches1;
    const int64_t i = pi * (256 >> P.cb) + r, j = pj * (1 << P.cb) + c;
    return (i < P.n0 && j < P.n1) ? i * P.n1 + j : -1;
}

// Cell of thread t in the warp-tile layout: a warp takes 4 x 8 cells (8 x 4
// in a patch of 4 columns), the warps row by row.
__device__ __forceinline__ void tile_cell(const PatchGrid& P, int t, int* r, int* c) {
    const int warp = t >> 5, lane = t & 31;
    if (P.cb < 3) {
        *r = 8 * warp + (lane >> 2);
        *c = lane & 3;
    } else {
        const int b = P.cb - 3;  // log2 of the warps in a row
        *r = 4 * (warp >> b) + (lane >> 3);
        *c = 8 * (warp & ((1 << b) - 1)) + (lane & 7);
    }
}


// How a stage is filled.
//  LOAD_SWIZZLED: tensor copies of boxes of 32 columns, swizzled.
//  LOAD_WIDE:     tensor copies of boxes of `pitch` columns, as they lie.
//  LOAD_RESIDUES: rows that are not whole 16-byte chunks, which no tensor map
//                 describes; but four rows are.  The stack is taken as groups
//                 of four rows (one tensor row each, the stack's last up to
//                 three rows left out), and the box rows r = k mod 4 come
//                 with one copy, from the place of row k in its group on:
//                 all of them start equally far, lead = (row * columns) & 3
//                 floats, from a 16-byte boundary of their slice, and slice z
//                 starts (z * n_in) & 3 floats from one.  A copy starts at
//                 that boundary, so cells lie lead floats further on in their
//                 row, and a whole slice its shift further.
constexpr int LOAD_SWIZZLED = 0, LOAD_WIDE = 1, LOAD_RESIDUES = 2;

// Where a box's cells lie in a slice's plane (unused fields 0).
struct BoxShape {
    int pitch;     // floats between rows (of one residue)
    int residues;  // LOAD_RESIDUES: floats between residues
};

// Box slot of input cell c.
template <int LOAD>
__device__ __forceinline__ int box_slot_of(int c, int2 org, FastDiv nd, BoxShape B) {
    const int row = (int)nd.div((uint32_t)c);
    const int r = row - org.x, cc = c - row * (int)nd.d - org.y;
    if constexpr (LOAD == LOAD_SWIZZLED) return r * PBOX_C + ((((cc >> 2) ^ (r & 7)) << 2) | (cc & 3));
    else if constexpr (LOAD == LOAD_WIDE) return r * B.pitch + cc;
    else return (r & 3) * B.residues + (r >> 2) * B.pitch + (int)((unsigned)row * nd.d & 3u) + cc;
}

// Whether a float32 is finite, from its exponent bits.
__device__ __forceinline__ bool finite_bits(float f) {
    return (__float_as_uint(f) & 0x7f800000u) != 0x7f800000u;
}

// Whether a float32 is normal (neither zero, subnormal, infinite nor NaN).
__device__ __forceinline__ bool normal_bits(unsigned u) {
    return (u & 0x7f800000u) - 0x00800000u < 0x7f000000u;
}

// widen() of a normal float32, from its bits: the double's high word is the
// sign, the exponent rebiased by 1023 - 127 and the top 20 fraction bits;
// the low word the last 3 fraction bits.
__device__ __forceinline__ double widen_normal(unsigned u) {
    const unsigned hi = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + ((1023u - 127u) << 20));
    return __hiloint2double((int)hi, (int)(u << 29));
}

// Accumulation modes of the TMA apply.
//  MODE_FAST:  float32 output, acc = fmaf(w, x, acc) with float32 weights in
//              the bank-aware gather order.
//  MODE_EXACT: the upstream float64 apply bit for bit (float32 input, float64
//              weights and output): every entry in stored (CSR) order as
//              acc = acc + w * (double)x with one rounding per operation, from 0.0.
//  MODE_FF:    float64 output from float-float arithmetic on the FP32 pipe
//              (the GB300 runs FP32 at 64x its FP64 rate): each weight as
//              hi + lo floats, each product x * hi split exactly into p + e
//              by an FMA (Dekker's product), the running sum kept as an
//              unevaluated pair (h, l) with Knuth's two-sum, and h + l added
//              in double once per output.  Entries in the gather order.
constexpr int MODE_FAST = 0, MODE_EXACT = 1, MODE_FF = 2;

// Longest row that MODE_FF sums as float pairs in a wide box.  With u = 2^-24
// and sums S of one sign, every product is off by at most 3 u^2 of its term, the
// rounding of err + r by u^2 (S + 2 of the term), and that of the k-th l by
// u |l| <= u^2 (k + 2) S: in all u^2 (n^2 / 2 + 3.5 n + 5) S, and 2^-53 S for the
// last addition, below 1e-12 S for n <= 20.  (Where roundings have one sign the
// bound is approached: 250 equal terms are off by 1e-12, 4,000 by 2.7e-10.)
// Longer rows are summed in float64, in stored order.  (Boxes of 32 swizzled
// columns hold patches whose rows have about 9 entries; their kernel tests
// nothing.)
constexpr int FF_ROW_MAX = 20;
// One in this many rows may be long; with more, the exact kernel takes the call.
// (2048^2 -> 819^2 rotated by 0.45, one row in 30 long, 1, 2, 4, 8, 16 slices:
// 97, 124, 189, 321, 587 us with the long rows here, 76 (gathered), 111, 178, 309,
// 568 exact; without long rows 52, 56, 72, 103, 168.)
constexpr int FF_LONG_SHARE = 64;

// Packed pairs of float32 (two slices of one output): the sm_100-family
// f32x2 instructions apply one IEEE operation, rounded to nearest, to both
// halves, at the issue cost of one scalar instruction.
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// One float-float step on a pair of slices: (h, l) += x * (wh + wl), with
// the weight given as the pairs wh, -wh and wl.  Per half the operations
// and their results are those of the scalar step
//     p = x wh;  e = fma(x, wh, -p);  r = fma(x, wl, e);
//     t = h + p;  bp = t - h;  err = (h - (t - bp)) + (p - bp);
//     h = t;  l = l + (err + r)
// (Dekker's product, Knuth's two-sum), written with pn = x (-wh) = -p so
// that no operand needs negating: fma(x, wh, pn) = x wh - p, h - pn = h + p,
// and p - bp = -(pn + bp), subtracted from h - (t - bp).  (The only
// difference is the sign of an exact zero p - bp, which cannot reach the
// sum: h - (t - bp) is never -0, as h starts at +0.)
__device__ __forceinline__ void ff_step2(uint64_t& h, uint64_t& l, uint64_t wh, uint64_t whn, uint64_t wl,
                                         uint64_t x) {
    const uint64_t pn = f2_mul(x, whn);
    const uint64_t e = f2_fma(x, wh, pn);
    const uint64_t r = f2_fma(x, wl, e);
    const uint64_t t = f2_sub(h, pn);
    const uint64_t bp = f2_sub(t, h);
    const uint64_t err = f2_sub(f2_sub(h, f2_sub(t, bp)), f2_add(pn, bp));
    h = t;
    l = f2_add(l, f2_add(err, r));
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ double as_double(float v) { return widen(v); }
__device__ __forceinline__ double as_double(double v) { return v; }

// TIN: the stack's type (double in the exact mode's wide boxes only; "floats"
// are cells then).
template <int SPS, int NST, int MINB, int MODE, int CT = CACHED_T, int LOAD = LOAD_SWIZZLED, int PL = PLANE,
          typename TIN = float>
__global__ void __launch_bounds__(32 * PATCH_WARPS, MINB)
    apply_patch_tma(const __grid_constant__ CUtensorMap tmap, const int64_t* __restrict__ row_ptr,
                    const int32_t* __restrict__ col, const uint16_t* __restrict__ slot,
                    const float* __restrict__ bval, const float* __restrict__ blo, const float* __restrict__ val,
                    const double* __restrict__ dval, double* __restrict__ vout64, FastDiv nd,
                    PatchGrid P, int64_t n_patches, const int2* __restrict__ origin, int BR, int stage_floats,
                    unsigned box_bytes, const TIN* __restrict__ vin, int64_t n_in, float* __restrict__ vout,
                    int64_t n_out, int64_t stack, int64_t chunk, unsigned* __restrict__ flags,
                    const uint8_t* __restrict__ perm, BoxShape box, const int2* __restrict__ extent) {
    constexpr bool EXACT = MODE == MODE_EXACT;
    constexpr bool OUT64 = MODE != MODE_FAST;
    // The float64-output modes give every slice of a stage its own 4 KB plane
    // (constant gather offsets; one box copy per slice) and let the last warp
    // done with a stage refill it.  The float32 mode, whose gathers are few
    // instructions, keeps one box copy per stage (slices packed BR rows
    // apart) and a producer thread that waits for the warps; measured faster
    // for it.
    constexpr bool PLANES = MODE != MODE_FAST || LOAD != LOAD_SWIZZLED;
    constexpr bool RESIDUES = LOAD == LOAD_RESIDUES;
    __shared__ __align__(8) uint64_t full[NST], empty[NST];
    __shared__ unsigned done[NST];  // warps done with each stage, counted over all its uses
    // entries CT .. CT + NX - 1 of every thread's row, read once per patch
    // (rows one or two entries longer than the registers hold are common;
    // reading those entries from global memory at every stage held back the
    // warp with the longest rows, and with it the stage's refill): their
    // slots, and their float32 weights (fast), float32 weight and rest
    // (compensated) or float64 weights (exact)
    // (boxes of more than 1536 cells come with coarse output cells: longer rows)
    constexpr int NX = CT > 0 ? (PL > 1536 ? 8 : MODE == MODE_FF ? FF_EXTRA : ROW_EXTRA) : 1;
    constexpr int NXF = MODE != MODE_EXACT ? NX : 1, NXL = MODE == MODE_FF ? NX : 1;
    constexpr int NXD = MODE == MODE_EXACT ? NX : 1;
    __shared__ uint16_t ex_slot[NX][32 * PATCH_WARPS];
    __shared__ float ex_hi[NXF][32 * PATCH_WARPS], ex_lo[NXL][32 * PATCH_WARPS];
    __shared__ double ex_d[NXD][32 * PATCH_WARPS];
    extern __shared__ __align__(1024) unsigned char ring_bytes[];
    TIN* ring = reinterpret_cast<TIN*>(ring_bytes);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int64_t p = blockIdx.x;
    // the thread's output: the warp tile layout, or for the exact and
    // compensated applies the patch's outputs by row length (a warp's lanes
    // then run chains of similar length)
    const int64_t d0 = (int64_t)blockIdx.y * chunk;
    const int64_t d1 = d0 + chunk < stack ? d0 + chunk : stack;
    const int2 org = origin[p];
    const int64_t ngroups = (d1 - d0 + SPS - 1) / SPS;
    // PLANES: one box copy per slice of the group (slices past the chunk are
    // not loaded); else one copy of box_bytes for the whole stage
    auto issue = [&](int st, int64_t grp) {
        const int64_t z0 = d0 + grp * SPS;
        if constexpr (PLANES) {
            const int n = (int)(d1 - z0 < SPS ? d1 - z0 : SPS);
            mbar_expect_tx(&full[st], (unsigned)n * box_bytes);
            for (int q = 0; q < n; q++)
                tma_load_3d(ring + (int64_t)st * stage_floats + q * PL, &tmap, org.y, org.x, (int)(z0 + q),
                            &full[st]);
        } else {
            mbar_expect_tx(&full[st], box_bytes);
            tma_load_3d(ring + (int64_t)st * stage_floats, &tmap, org.y, org.x, (int)z0, &full[st]);
        }
    };
    // LOAD_RESIDUES: one lane per copy, n slices of four each.  Where the
    // footprint reaches the stack's rows after its last group of four, the
    // warp's lanes bring the stage's cells themselves.
    auto slice_shift = [&](int64_t z) { return (int)((unsigned)z * (unsigned)n_in & 3u); };
    const int2 ext = RESIDUES && org.x >= 0 ? extent[p] : make_int2(0, 0);
    const int64_t in_rows = RESIDUES ? n_in / nd.d : 0;  // of a slice
    auto issue_residues = [&](int st, int64_t grp) {
        const int64_t z0 = d0 + grp * SPS;
        const int n = (int)(d1 - z0 < SPS ? d1 - z0 : SPS);
        TIN* stage = ring + (int64_t)st * stage_floats;
        if (z0 + n == stack && (stack - 1) * in_rows + org.x + ext.x > (stack * in_rows & ~(int64_t)3)) {
            for (int q = 0; q < n; q++)
                for (int r = 0; r < ext.x; r++) {
                    const unsigned row = (unsigned)(org.x + r);
                    const int lead = (int)(row * nd.d & 3u);
                    TIN* dst = stage + q * PL + (r & 3) * box.residues + (r >> 2) * box.pitch +
                                 slice_shift(z0 + q);
                    const TIN* src = vin + (z0 + q) * n_in + (int64_t)row * nd.d + org.y - lead;
                    const int cells = ext.y + lead;
                    for (int c = lane; c < cells; c += 32) dst[c] = __ldg(src + c);
                }
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[st]);
            return;
        }
        if (lane == 0) mbar_expect_tx(&full[st], (unsigned)n * 4u * box_bytes);
        __syncwarp();
        for (int l = lane; l < 4 * n; l += 32) {
            const int q = l >> 2, k = l & 3;
            const int64_t row = (z0 + q) * in_rows + org.x + k;  // of the stack
            const int lead = (int)((unsigned)(org.x + k) * nd.d & 3u) + slice_shift(z0 + q);
            tma_load_2d(stage + q * PL + k * box.residues, &tmap, (int)(row & 3) * (int)nd.d + org.y - lead, (int)(row >> 2),
                        &full[st]);
        }
    };
    // the first stages' copies start before the threads fetch their rows, so
    // that the copies and the row fetches overlap (the barriers are ready for
    // the other threads after the __syncthreads below)
    if (org.x >= 0 && t == 0) {
        for (int k = 0; k < NST; k++) {
            mbar_init(&full[k], 1);
            mbar_init(&empty[k], PATCH_WARPS);
            done[k] = 0u;
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if constexpr (!RESIDUES)
            for (int k = 0; k < NST && k < ngroups; k++) issue(k, k);
    }
    if constexpr (RESIDUES) {
        if (org.x >= 0 && warp == 0) {
            __syncwarp();
            for (int k = 0; k < NST && k < ngroups; k++) issue_residues(k, k);
        }
    }
    int pr, pc;
    tile_cell(P, t, &pr, &pc);
    if (OUT64 && perm) {
        const int raw = perm[p * (32 * PATCH_WARPS) + t];
        pr = raw >> P.cb;
        pc = raw & ((1 << P.cb) - 1);
    }
    const int64_t o = patch_cell(P, p, pr, pc);
    int64_t s = 0, e = 0;
    if (o >= 0) {
        s = row_ptr[o];
        e = row_ptr[o + 1];
    }
    const int nk = (int)(e - s);
    float* out = vout + (o >= 0 ? o : 0);
    if (org.x < 0) {
        // no entries (all zeros) or a footprint larger than the box: the whole block
        if (o >= 0) {
            if constexpr (OUT64) {
                for (int64_t d = d0; d < d1; d++) {
                    const TIN* a = vin + d * n_in;
                    double acc = 0.0;
                    for (int64_t k = s; k < e; k++) acc = __dadd_rn(acc, __dmul_rn(dval[k], (double)__ldg(a + col[k])));
                    vout64[d * n_out + o] = acc;
                }
            } else if constexpr (sizeof(TIN) == 4) {
                apply_direct(s, e, col, val, vin, n_in, out, n_out, d0, d1);
            }
        }
        return;
    }
    // The compensated apply runs every lane of a warp to the warp's longest
    // row (a uniform bound, no divergent branch per entry).  A lane's entries
    // past its own row have zero weights and slot 0: such a step leaves the
    // pair (h, l) unchanged for a finite input word; a non-finite one makes
    // the sum NaN, which sends that output and slice to the exact loop.
    // a long row's lane takes no float-float step: its entries here are none
    const bool long_row = MODE == MODE_FF && LOAD != LOAD_SWIZZLED && nk > FF_ROW_MAX;
    const int nf = long_row ? 0 : nk;
    // (written so: with s + nf the swizzled kernel of six slices takes 80 registers
    // for 64, 577 us for 573, and with a choice of s and e the wide ones 617 for 600)
    const int64_t ef = LOAD == LOAD_SWIZZLED ? e : s + nf;
    const int kwarp = MODE == MODE_FF ? __reduce_max_sync(0xffffffffu, nf) : nk;
    // PLANES: every slice of a stage has its own 4 KB plane, 1024-byte
    // aligned, so all slices see the same swizzle phase and a gather's
    // slices differ by constant offsets.  Otherwise the rows of slice q start
    // at row q * BR of the swizzle pattern: with BR a multiple of 4, odd
    // slices see the pattern shifted by 4 rows, which is the chunk index
    // xor 4 (slot xor 16).
    const int plane = PLANES ? PL : BR * PBOX_C;
    const int flip = PLANES ? 0 : ((BR & 4) ? 16 : 0);
    // (CT = 0 keeps a single dummy slot: every entry is read from memory)
    int li[CT > 0 ? CT : 1];
    float w[CT > 0 ? CT : 1];
    double wd[CT > 0 ? CT : 1];
    // the compensated mode's weights as packed pairs (wh, wh), (-wh, -wh), (wl, wl)
    uint64_t fh[CT > 0 ? CT : 1], fhn[CT > 0 ? CT : 1], fl[CT > 0 ? CT : 1];
#pragma unroll
    for (int k = 0; k < CT; k++) {
        if constexpr (EXACT) {
            li[k] = k < nk ? box_slot_of<LOAD>(col[s + k], org, nd, box) : 0;
            wd[k] = k < nk ? dval[s + k] : 0.0;
            w[k] = 0.f;
        } else if constexpr (MODE == MODE_FF) {
            li[k] = k < nf ? (int)slot[s + k] : 0;
            const float a = k < nf ? bval[s + k] : 0.f, b = k < nf ? blo[s + k] : 0.f;
            fh[k] = f2_pack(a, a);
            fhn[k] = f2_pack(-a, -a);
            fl[k] = f2_pack(b, b);
        } else {
            li[k] = k < nk ? (int)slot[s + k] : 0;
            w[k] = k < nk ? bval[s + k] : 0.f;
            wd[k] = 0.0;
        }
    }
    if constexpr (CT > 0) {
#pragma unroll
        for (int j = 0; j < NX; j++) {
            const bool has = CT + j < nf;
            if constexpr (EXACT) {
                ex_slot[j][t] = has ? (uint16_t)box_slot_of<LOAD>(col[s + CT + j], org, nd, box) : (uint16_t)0;
                ex_d[j][t] = has ? dval[s + CT + j] : 0.0;
            } else {
                ex_slot[j][t] = has ? slot[s + CT + j] : (uint16_t)0;
                ex_hi[j][t] = has ? bval[s + CT + j] : 0.f;
                if constexpr (MODE == MODE_FF) ex_lo[j][t] = has ? blo[s + CT + j] : 0.f;
            }
        }
    }
    __syncthreads();
    for (int64_t grp = 0; grp < ngroups; grp++) {
        const int st = (int)(grp % NST);
        const unsigned ph = (unsigned)((grp / NST) & 1);
        const bool got = mbar_wait_bounded(&full[st], ph);
        if (!__all_sync(0xffffffffu, got)) {
            if (lane == 0) {
                atomicOr(flags, FLAG_TIMEOUT);
                // copies of this block that may still be in flight: bounded wait before leaving
                for (int64_t q = grp + 1; q < grp + NST && q < ngroups; q++)
                    (void)mbar_wait_bounded(&full[q % NST], (unsigned)((q / NST) & 1));
            }
            return;
        }
        const TIN* buf = ring + (int64_t)st * stage_floats;
        const int64_t ds = d0 + grp * SPS;
        int off[SPS];  // the slices' planes in the stage
#pragma unroll
        for (int q = 0; q < SPS; q++) off[q] = q * plane + (RESIDUES ? slice_shift(ds + q) : 0);
        auto cell_of = [&](int q, int slot) { return buf[off[q] + (slot ^ ((q & 1) ? flip : 0))]; };
        if constexpr (EXACT) {
            if (o >= 0) {
                double acc[SPS];
#pragma unroll
                for (int q = 0; q < SPS; q++) acc[q] = 0.0;
#pragma unroll
                for (int k = 0; k < CT; k++) {
                    if (k < nk) {
#pragma unroll
                        for (int q = 0; q < SPS; q++)
                            acc[q] = __dadd_rn(
                                acc[q], __dmul_rn(wd[k], as_double(cell_of(q, li[k]))));
                    }
                }
                if constexpr (CT > 0) {
#pragma unroll
                    for (int j = 0; j < NX; j++) {
                        if (CT + j < nk) {
                            const double wk = ex_d[j][t];
                            const int sk = ex_slot[j][t];
#pragma unroll
                            for (int q = 0; q < SPS; q++)
                                acc[q] = __dadd_rn(acc[q],
                                                   __dmul_rn(wk, as_double(cell_of(q, sk))));
                        }
                    }
                }
                for (int64_t k = s + (CT > 0 ? CT + NX : 0); k < e; k++) {
                    const double wk = dval[k];
                    const int sk = box_slot_of<LOAD>(col[k], org, nd, box);
#pragma unroll
                    for (int q = 0; q < SPS; q++)
                        acc[q] = __dadd_rn(acc[q], __dmul_rn(wk, as_double(cell_of(q, sk))));
                }
#pragma unroll
                for (int q = 0; q < SPS; q++)
                    if (ds + q < d1) vout64[(ds + q) * n_out + o] = acc[q];
            }
        } else if constexpr (MODE == MODE_FF) {
            if (o >= 0) {
                // slices 2j and 2j + 1 of the stage as one packed pair
                static_assert(SPS % 2 == 0, "the compensated apply stages slices in pairs");
                uint64_t h2[SPS / 2], l2[SPS / 2];
#pragma unroll
                for (int j = 0; j < SPS / 2; j++) h2[j] = l2[j] = 0ull;
#pragma unroll
                for (int k = 0; k < CT; k++) {
                    if (k < kwarp) {
                        const int a = li[k];
#pragma unroll
                        for (int j = 0; j < SPS / 2; j++)
                            ff_step2(h2[j], l2[j], fh[k], fhn[k], fl[k],
                                     f2_pack(cell_of(2 * j, a), cell_of(2 * j + 1, a)));
                    }
                }
                if constexpr (CT > 0) {
#pragma unroll
                    for (int j = 0; j < NX; j++) {
                        if (CT + j < kwarp) {
                            const float wk = ex_hi[j][t], wlk = ex_lo[j][t];
                            const uint64_t kh = f2_pack(wk, wk), khn = f2_pack(-wk, -wk), kl = f2_pack(wlk, wlk);
                            const int a = ex_slot[j][t];
#pragma unroll
                            for (int q = 0; q < SPS / 2; q++)
                                ff_step2(h2[q], l2[q], kh, khn, kl,
                                         f2_pack(cell_of(2 * q, a), cell_of(2 * q + 1, a)));
                        }
                    }
                }
                for (int64_t k = s + (CT > 0 ? CT + NX : 0); k < ef; k++) {
                    const float wk = bval[k], wlk = blo[k];
                    const uint64_t kh = f2_pack(wk, wk), khn = f2_pack(-wk, -wk), kl = f2_pack(wlk, wlk);
                    const int a = slot[k];
#pragma unroll
                    for (int j = 0; j < SPS / 2; j++)
                        ff_step2(h2[j], l2[j], kh, khn, kl,
                                 f2_pack(cell_of(2 * j, a), cell_of(2 * j + 1, a)));
                }
                float h[SPS], l[SPS];
#pragma unroll
                for (int j = 0; j < SPS / 2; j++) {
                    const float2 hv = f2_unpack(h2[j]), lv = f2_unpack(l2[j]);
                    h[2 * j] = hv.x;
                    h[2 * j + 1] = hv.y;
                    l[2 * j] = lv.x;
                    l[2 * j + 1] = lv.y;
                }
                // The usual stage (every slice in range, every h and l a
                // normal float) is tested once, with bitwise ands and a single
                // branch, and stored without further tests (per-slice tests
                // and branches were a measured share of the instruction
                // stream).  Anything else takes the per-slice path.
                bool usual = ds + SPS <= d1 && !long_row;
#pragma unroll
                for (int q = 0; q < SPS; q++)
                    usual = usual & normal_bits(__float_as_uint(h[q])) & normal_bits(__float_as_uint(l[q]));
                if (usual) {
                    double* dst = vout64 + ds * n_out + o;
#pragma unroll
                    for (int q = 0; q < SPS; q++)
                        dst[q * n_out] =
                            __dadd_rn(widen_normal(__float_as_uint(h[q])), widen_normal(__float_as_uint(l[q])));
                } else {
#pragma unroll
                    for (int q = 0; q < SPS; q++) {
                        if (ds + q >= d1) continue;
                        double r;
                        const unsigned uh = __float_as_uint(h[q]), ul = __float_as_uint(l[q]);
                        if (normal_bits(uh) && normal_bits(ul)) {
                            r = __dadd_rn(widen_normal(uh), widen_normal(ul));
                        } else if (nk == 0) {
                            r = 0.0;
                        } else if (!long_row && finite_bits(h[q]) && finite_bits(l[q])) {
                            r = __dadd_rn(widen(h[q]), widen(l[q]));
                        } else {
                            // a long row, or a float32 partial sum overflowed,
                            // or an input or a weight is not finite (or a padded
                            // step read a non-finite word): this output and slice
                            // in float64, stored order (the exact apply's sum)
                            r = 0.0;
                            for (int64_t k = s; k < e; k++)
                                r = __dadd_rn(r, __dmul_rn(dval[k], as_double(cell_of(q, box_slot_of<LOAD>(col[k], org, nd, box)))));
                        }
                        vout64[(ds + q) * n_out + o] = r;
                    }
                }
            }
        } else if (o >= 0) {
            float acc[SPS];
#pragma unroll
            for (int q = 0; q < SPS; q++) acc[q] = 0.f;
#pragma unroll
            for (int k = 0; k < CT; k++) {
                if (k < nk) {
#pragma unroll
                    for (int q = 0; q < SPS; q++)
                        acc[q] = fmaf(w[k], cell_of(q, li[k]), acc[q]);
                }
            }
            if constexpr (CT > 0) {
#pragma unroll
                for (int j = 0; j < NX; j++) {
                    if (CT + j < nk) {
                        const float wk = ex_hi[j][t];
                        const int sk = ex_slot[j][t];
#pragma unroll
                        for (int q = 0; q < SPS; q++)
                            acc[q] = fmaf(wk, cell_of(q, sk), acc[q]);
                    }
                }
            }
            for (int64_t k = s + (CT > 0 ? CT + NX : 0); k < e; k++) {
                const float wk = bval[k];
                const int sk = slot[k];
#pragma unroll
                for (int q = 0; q < SPS; q++) acc[q] = fmaf(wk, cell_of(q, sk), acc[q]);
            }
#pragma unroll
            for (int q = 0; q < SPS; q++)
                if (ds + q < d1) out[(ds + q) * n_out] = acc[q];
        }
        // The last warp done with the stage refills it, so no warp waits for
        // the others (the slowest warp, with the longest rows, no longer
        // holds a producer thread back).  Its lanes' reads of the stage are
        // ordered before the count (syncwarp, then a release fence); the last
        // one acquires them all before the async-proxy copy overwrites it.
        __syncwarp();
        if constexpr (RESIDUES) {
            unsigned last = 0u;
            if (lane == 0) {
                __threadfence_block();
                last = atomicAdd(&done[st], 1u) + 1u == (unsigned)(grp / NST + 1) * PATCH_WARPS;
                if (last) {
                    __threadfence_block();
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                }
            }
            last = __shfl_sync(0xffffffffu, last, 0);
            __syncwarp();
            if (last && grp + NST < ngroups) issue_residues(st, grp + NST);
        } else if constexpr (PLANES) {
            if (lane == 0) {
                __threadfence_block();
                const unsigned n = atomicAdd(&done[st], 1u) + 1u;
                if (n == (unsigned)(grp / NST + 1) * PATCH_WARPS && grp + NST < ngroups) {
                    __threadfence_block();
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    issue(st, grp + NST);
                }
            }
        } else {
            if (lane == 0) mbar_arrive(&empty[st]);  // this warp is done with the stage
            if (t == 0 && grp + NST < ngroups) {
                if (!mbar_wait_bounded(&empty[st], ph)) {
                    atomicOr(flags, FLAG_TIMEOUT);
                    for (int64_t q = grp + 1; q < grp + NST && q < ngroups; q++)
                        (void)mbar_wait_bounded(&full[q % NST], (unsigned)((q / NST) & 1));
                    return;
                }
                // the warps' generic-proxy reads of the stage before the async-proxy writes
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                issue(st, grp + NST);
            }
        }
    }
}

}  // namespace
}  // namespace rg
