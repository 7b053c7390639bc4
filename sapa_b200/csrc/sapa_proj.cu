// sapa_proj.cu — the step in front of the attention: GroupNorm followed by the 1x1 query / key projection
// (reference: sapa_base.py:27-34, sapa_deform.py:35-42), as ONE dense GEMM per image on the 5th-generation tensor cores.
//
// GroupNorm is affine per (image, channel) once the group statistics are known, so it folds into the projection:
//   out[b, j, p] = sum_c W[j, c] * (gamma_c * rstd_bg * (x[b, c, p] - mean_bg) + beta_c) + bias_j
//                = sum_c W'[b, j, c] * x[b, c, p] + bias'[b, j]
//   W'[b, j, c]  = W[j, c] * gamma_c * rstd_bg(c),      bias'[b, j] = bias_j + sum_c W[j, c] * (beta_c - mean_bg(c) * gamma_c * rstd_bg(c))
// Three launches: (1) partial sums of x and x^2 per (image, group) - one pass over x at memory speed, float64 partials;
// (2) the fold above (tiny); (3) a persistent GEMM kernel that reads x exactly once more and writes out.  The normalised
// activation tensor of the unfused sequence (one write + one read of the size of x) never exists.
//
// The launches take a LIST of problems: all projections of a module share them, and what a problem does not need is left out
// (16-bit rows without a norm are multiplied with the weight as it is: no statistics, no fold).  A launch of a small problem is
// latency: the four GEMMs and four folds of a SAPADeform module (4 x 256 x 32x32, d = 128, 288 offset rows, float16) took 41 us and
// the gaps between them, their one launch takes 13 (the module 91 -> 42 us); three chained SAPA modules (16 x 256, 16x16 -> 128x128,
// bfloat16), eighteen launches before, 293 -> 220 us.
//
// GEMM kernel (tcgen05 / TMEM; one CTA per SM, 128-pixel tiles):
//   D[128 px x d] (+)= A[128 px x k] * B[k x d],  A = x^T, B = W' (K-major: channels contiguous)
//   * warp 4 (one lane): TMA producer of the activations, warp 6 (one lane): TMA producer of the W' blocks.  A stage =
//     128 px x (128 B / esize) channels of x as boxes of one 128-byte pixel row per channel (128-byte swizzle) plus the
//     matching d x 128 B block of W' (canonical K-major layout).
//   * 16-bit types: the landed boxes ARE the canonical operand layout for an operand whose M dimension is the contiguous
//     one ("MN-major"), and the tensor core reads them in place.
//   * float32, warps 7-14: 3xTF32 split AND transposition.  The tensor core reads tf32 (the upper 19 bits); the product
//     is evaluated as hi*hi + lo*hi + hi*lo with hi = x & 0xffffe000, lo = x - hi (exact): float32 accuracy (1e-6).  The
//     warps read a landed ring slot (lane = channel, 16 bytes = 4 pixels) and write hi and lo into an operand slot as
//     K-major rows (row = pixel, 128 bytes = the stage's 32 channels, 128-byte swizzle): both sides are free of bank
//     conflicts and the ring slot is released at once.  (The landed boxes can also be fed as an MN-major tf32 operand:
//     that needs the 128-byte swizzle of 32-byte chunks - CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, descriptor layout type 1,
//     4-row atoms; with the ordinary swizzle the product is wrong.  That form is as accurate and no faster.)  W' arrives
//     already split.
//   * warp 5: issues tcgen05.mma (M = 128, N = d, K = 32 bytes) into one of two TMEM accumulators, frees a stage with
//     tcgen05.commit, signals the epilogue with another commit.  The whole warp runs the loop, so that descriptors stay in uniform
//     registers (tc_mma: an instruction from a branch of one lane took 57 clocks; q of 16 x 256 x 128x128, d = 128, bfloat16 84 -> 78 us,
//     the three lists of the chain above 57 -> 52); for float32 with d <= 128 the terms x_hi * W'_hi and x_hi * W'_lo are ONE
//     instruction of N = 2d (the two W' blocks are adjacent rows of the operand; the epilogue adds the two halves of the
//     accumulator): 8 instead of 12 MMAs per stage.
//   * warps 0-3: epilogue.  tcgen05.ld (lane = pixel, column = output channel), add bias', store: for a fixed output
//     channel the 32 lanes of a warp write 32 consecutive pixels.  Runs under the MMAs of the next tile.
// Tiles walk the images from the last to the first: the statistics pass has just read them in ascending order, so the
// tail of x is what the L2 still holds.
// Every mbarrier wait is bounded; a wait that gives up raises g_wait_timeout and the CTA drains and frees its TMEM.
#include "umma_util.cuh"

#include <algorithm>
#include <cstdint>
#include <type_traits>

namespace sapa {

namespace proj {

using namespace tmau;
using namespace ummau;

constexpr int TILE_PX = 128;
constexpr int EPI_WARPS = 4, TMA_WARP = 4, MMA_WARP = 5, W_WARP = 6, SPLIT_WARP0 = 7, SPLIT_WARPS = 8;
constexpr int THREADS = (SPLIT_WARP0 + SPLIT_WARPS) * 32;
constexpr int Y_STAGE = 16384;           // bytes of activations per stage: 128 px x (128 B / esize) channels
constexpr int MAX_SLOTS = 8;              // slots per ring
constexpr int OP_SLOTS_F32 = 2, OP_SLOTS_16 = 4;     // operand ring depth (the kernel is not sensitive to it)
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int STAT_THREADS = 256, MAX_SPLIT = 64, MAX_GROUPS = 256;
constexpr int FOLD_ROWS = STAT_THREADS / 32; // rows of W' per block of the fold
constexpr int MAX_PROBLEMS = 6;              // of one launch: parts of up to 256 output rows
constexpr int MAX_LIST = 3;                  // projections of a call
constexpr long long STAT_SLICE = 32768;      // bytes

__device__ int g_wait_timeout = 0;

struct Problem {
    CUtensorMap x_map;              // (pixel, channel, 1, image), box = one 128-byte pixel row x (128 B / esize) channels
    CUtensorMap whi_map, wlo_map;   // (channel, output channel, 1, image), box = 128 bytes of channels x d rows
    const float *bias;              // folded bias [images or 1][d]; nullptr: `bias_as_given`
    const void *bias_as_given;      // [d] of the activations' type on a 16-byte boundary, or nullptr (no bias)
    void *out;                      // first of the d rows of image 0; images are out_rows rows of HW elements apart
    int out_rows;
    int shuffle_w;                  // > 0: the rows are sub-pixels, written as torch.pixel_shuffle(., 2) would place them (row
                                    // 4o + 2i + j of an image of this width = pixels (2y + i, 2x + j) of channel o)
    int B, HW, d, w_per_image, tiles_per_image, kblocks;
    int wide;                       // float32: hi*hi and hi*lo in ONE instruction of N = 2d (W' hi and lo blocks are adjacent rows)
    int tiles_end;                  // tiles of the problems up to and including this one
};
struct Args {
    Problem p[MAX_PROBLEMS];
    int count, total_tiles;
    int w_rows;                     // largest d of the list: what an operand slot is laid out for
    int nx, no, tmem_cols, acc_cols;
};
// where a tile of the list lies
struct TileAt { int b, px0; };
__device__ __forceinline__ const Problem &find_tile(const Args &a, int tile, TileAt &at) {
    int i = 0;
    while (i + 1 < a.count && tile >= a.p[i].tiles_end) ++i;
    const Problem &p = a.p[i];
    const int local = tile - (i > 0 ? a.p[i - 1].tiles_end : 0), bi = local / p.tiles_per_image;
    at.b = p.B - 1 - bi;
    at.px0 = (local - bi * p.tiles_per_image) * TILE_PX;
    return p;
}

// Shared-memory matrix descriptor (64 bits).  Low word: start address (bits 0-13) and leading byte offset (bits 16-29),
// both in 16-byte units.  High word: stride byte offset in 16-byte units (bits 0-13 = descriptor bits 32-45), descriptor
// version 1 (bit 14 = bit 46), layout type 2 = 128-byte swizzle of 16-byte chunks (bits 29-31 = bits 61-63; 8-row atoms
// of 1 KB, aligned to 1 KB).  Every operand of this kernel has a stride of 1 KB between its 8-row atoms, so they all
// share one high word.  (Layout type 1, the 128-byte swizzle of 32-byte chunks with 4-row atoms, is what a tf32 operand
// needs when its M / N dimension is the contiguous one; it is not used any more, see the header.)
constexpr unsigned DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void store_out(float *p, float v) { __stcs(p, v); }
__device__ __forceinline__ void store_out(__half *p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void store_out(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

// ---------------------------------------------------------------------------------- the GEMM kernel
// Shared memory: an activation ring (NX slots of 16 KB, filled by TMA) and an operand ring (NO slots).  16-bit types:
// the tensor core reads the activations straight from their ring slot and an operand slot holds only the W' block.
// float32: an operand slot holds the split activations (hi, lo) and the W' blocks (hi, lo); the split warps move a
// landed slot into it and hand the ring slot back at once, so the loads in flight do not wait for the MMAs.
// TO = type of the output (that of x, or 16 bits of a float32 product)
template <typename T, typename TO>
__global__ void __launch_bounds__(THREADS, 1) sapa_proj_umma_kernel(const __grid_constant__ Args a) {
    constexpr bool F32 = sizeof(T) == 4;
    constexpr int KCH = 128 / (int)sizeof(T);        // channels per stage = one 128-byte row of the weight block
    constexpr int PXG = 128 / (int)sizeof(T);        // pixels per activation box = one 128-byte row
    constexpr int NBOX = TILE_PX / PXG;
    constexpr int KSTEPS = 4;                        // one tcgen05.mma covers 32 bytes of channels: 8 (tf32) or 16 (16-bit)
    constexpr unsigned A_BOX = KCH * 128;            // bytes of one activation box = distance between 128-byte pixel groups
    constexpr unsigned A_KSTEP = A_BOX / KSTEPS;     // KCH / 4 channels further down the box
    // activation operand: 16-bit types are read where TMA put them (pixels contiguous, 8-channel atoms, 128-byte swizzle);
    // float32 is rewritten by the split warps as K-major rows (one pixel = 128 bytes of channels, 8-pixel atoms)

    extern __shared__ unsigned char smem_dyn[];
    const unsigned xring = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned nx = (unsigned)a.nx, no = (unsigned)a.no;
    const unsigned w_ofs = F32 ? 2u * Y_STAGE : 0u;                       // W' blocks inside an operand slot: d x 128 bytes (float32: hi, then lo)
    const unsigned op_bytes = w_ofs + (F32 ? 2u : 1u) * (unsigned)a.w_rows * 128u;
    const unsigned opring = xring + nx * (unsigned)Y_STAGE;
    const unsigned bars = opring + no * op_bytes;
    const unsigned xfull0 = bars, xempty0 = bars + 8 * MAX_SLOTS, ready0 = bars + 16 * MAX_SLOTS, wfull0 = bars + 24 * MAX_SLOTS;
    const unsigned oempty0 = bars + 32 * MAX_SLOTS, tfull0 = bars + 40 * MAX_SLOTS, tempty0 = tfull0 + 16, tmem_slot = tempty0 + 16;

    const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
    if (tid == 0) {
        for (unsigned i = 0; i < nx; ++i) {
            mbar_init(xfull0 + 8 * i, 1);
            mbar_init(xempty0 + 8 * i, F32 ? SPLIT_WARPS * 32 : 1);
        }
        for (unsigned i = 0; i < no; ++i) {
            mbar_init(ready0 + 8 * i, SPLIT_WARPS * 32);
            mbar_init(wfull0 + 8 * i, 1);
            mbar_init(oempty0 + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(tfull0 + 8 * i, 1);
            mbar_init(tempty0 + 8 * i, EPI_WARPS * 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == MMA_WARP) {            // the whole warp allocates the accumulator columns
        tc_alloc(tmem_slot, (unsigned)a.tmem_cols);
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    begin_after_previous();
    tc_fence_after();
    unsigned tmem_base;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(tmem_base) : "r"(tmem_slot) : "memory");
    tmem_base = warp_uniform(tmem_base);

    const unsigned acc_cols = (unsigned)a.acc_cols;       // accumulator columns per tile
    bool ok = true;

    if (warp == TMA_WARP) {            // activations: global -> ring
        if (lane == 0) {
            unsigned it = 0;
            for (int tile = blockIdx.x; tile < a.total_tiles && ok; tile += gridDim.x) {
                TileAt at;
                const Problem &p = find_tile(a, tile, at);
                for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
                    const unsigned r = it % nx, rph = (it / nx) & 1u;
                    if (!mbar_wait_bounded(xempty0 + 8 * r, rph ^ 1u)) { ok = false; break; }
                    const unsigned slot = xring + r * (unsigned)Y_STAGE, full = xfull0 + 8 * r;
                    mbar_expect_tx(full, Y_STAGE);
#pragma unroll
                    for (int j = 0; j < NBOX; ++j) tma_load_4d(slot + j * A_BOX, &p.x_map, full, at.px0 + j * PXG, kb * KCH, 0, at.b);
                }
            }
        }
    } else if (warp == W_WARP) {       // W' blocks: global (L2 resident) -> operand ring
        if (lane == 0) {
            unsigned it = 0;
            for (int tile = blockIdx.x; tile < a.total_tiles && ok; tile += gridDim.x) {
                TileAt at;
                const Problem &p = find_tile(a, tile, at);
                const int wb = p.w_per_image ? at.b : 0;
                const unsigned w_bytes = (unsigned)p.d * 128u;
                for (int kb = 0; kb < p.kblocks; ++kb, ++it) {
                    const unsigned o = it % no, oph = (it / no) & 1u;
                    if (!mbar_wait_bounded(oempty0 + 8 * o, oph ^ 1u)) { ok = false; break; }
                    const unsigned slot = opring + o * op_bytes + w_ofs, full = wfull0 + 8 * o;
                    mbar_expect_tx(full, (int)((F32 ? 2u : 1u) * w_bytes));
                    tma_load_4d(slot, &p.whi_map, full, kb * KCH, 0, 0, wb);
                    if (F32) tma_load_4d(slot + w_bytes, &p.wlo_map, full, kb * KCH, 0, 0, wb);
                }
            }
        }
    } else if (warp == MMA_WARP) {     // the whole warp, one lane issues (tc_mma)
        const unsigned idesc0 = (1u << 4) | (UmmaFormat<T>::code << 7) | (UmmaFormat<T>::code << 10) | (F32 ? 0u : (1u << 15)) | ((unsigned)(TILE_PX >> 4) << 24);
        const unsigned leader = elect_leader();
        // low descriptor words per ring slot are base + slot * pitch; a K step adds a constant (all in 16-byte units)
        const unsigned a_base = warp_uniform(F32 ? desc_lo(opring, 16) : desc_lo(xring, A_BOX));
        const unsigned a_pitch = (F32 ? op_bytes : (unsigned)Y_STAGE) >> 4, a_kstep = (F32 ? 32u : A_KSTEP) >> 4;
        const unsigned b_base = warp_uniform(desc_lo(opring + w_ofs, 16)), b_pitch = op_bytes >> 4;
        unsigned r = 0, rph = 0, o = 0, oph = 0, ti = 0;
        for (int tile = blockIdx.x; tile < a.total_tiles && ok; tile += gridDim.x, ++ti) {
            const unsigned buf = ti & 1u, tph = (ti >> 1) & 1u;
            TileAt at;
            const Problem &p = find_tile(a, tile, at);
            const int kblocks = p.kblocks;
            const unsigned w_bytes = (unsigned)p.d * 128u, wide = F32 ? (unsigned)p.wide : 0u;
            const unsigned idesc = idesc0 | idesc_n((unsigned)p.d), idesc_wide = idesc0 | idesc_n(2u * (unsigned)p.d);      // N = d, 2d
            ok = mbar_wait_warp(tempty0 + 8 * buf, tph ^ 1u);
            if (!ok) break;
            tc_fence_after();
            const unsigned d_tmem = tmem_base + buf * acc_cols;
            for (int kb = 0; kb < kblocks; ++kb) {
                ok = mbar_wait_warp((F32 ? ready0 + 8 * o : xfull0 + 8 * r), F32 ? oph : rph) && mbar_wait_warp(wfull0 + 8 * o, oph);
                if (!ok) break;
                tc_fence_after();
                const unsigned a0 = a_base + (F32 ? o : r) * a_pitch, b0 = b_base + o * b_pitch;
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks) {
                    const unsigned first = (ks != 0 || kb != 0) ? 1u : 0u;
                    if (F32 && wide) {
                        // x_hi * [W'_hi ; W'_lo] as one instruction of N = 2d (columns [0, d) and [d, 2d) of the
                        // accumulator, added by the epilogue), then x_lo * W'_hi into the first half
                        tc_mma<F32>(leader, d_tmem, a0 + ks * a_kstep, b0 + ks * 2u, DESC_HI, idesc_wide, first);
                        tc_mma<F32>(leader, d_tmem, a0 + (Y_STAGE >> 4) + ks * a_kstep, b0 + ks * 2u, DESC_HI, idesc, 1u);
                    } else {
                        tc_mma<F32>(leader, d_tmem, a0 + ks * a_kstep, b0 + ks * 2u, DESC_HI, idesc, first);
                        if (F32) {
                            tc_mma<F32>(leader, d_tmem, a0 + (Y_STAGE >> 4) + ks * a_kstep, b0 + ks * 2u, DESC_HI, idesc, 1u);      // lo * hi
                            tc_mma<F32>(leader, d_tmem, a0 + ks * a_kstep, b0 + (w_bytes >> 4) + ks * 2u, DESC_HI, idesc, 1u);      // hi * lo
                        }
                    }
                }
                if (!F32) tc_commit_by(leader, xempty0 + 8 * r);   // the activation slot is free once these MMAs have read it
                tc_commit_by(leader, oempty0 + 8 * o);             // and so is the operand slot
                if (++r == nx) { r = 0; rph ^= 1u; }
                if (++o == no) { o = 0; oph ^= 1u; }
            }
            if (ok) tc_commit_by(leader, tfull0 + 8 * buf);        // the accumulator is complete once all MMAs so far are done
        }
    } else if (warp >= SPLIT_WARP0) {
        if (F32) {
            const int st = tid - SPLIT_WARP0 * 32;
            unsigned it = 0;
            for (int tile = blockIdx.x; tile < a.total_tiles && ok; tile += gridDim.x) {
                TileAt at;
                const int kblocks = find_tile(a, tile, at).kblocks;
                for (int kb = 0; kb < kblocks; ++kb, ++it) {
                    const unsigned r = it % nx, rph = (it / nx) & 1u, o = it % no, oph = (it / no) & 1u;
                    if (!mbar_wait_bounded(xfull0 + 8 * r, rph) || !mbar_wait_bounded(oempty0 + 8 * o, oph ^ 1u)) { ok = false; break; }
                    const unsigned src = xring + r * (unsigned)Y_STAGE, dst = opring + o * op_bytes;
                    // item = (pixel group j, channel c = lane, 16-byte chunk q = 4 pixels): two warps per pixel group
                    const int sw = st >> 5, c = st & 31, j = sw >> 1;
                    unsigned v[4][4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {            // all four loads in flight before the first store
                        const int q = (sw & 1) * 4 + i;
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[i][0]), "=r"(v[i][1]), "=r"(v[i][2]), "=r"(v[i][3])
                                     : "r"(src + (unsigned)j * A_BOX + (unsigned)c * 128u + (unsigned)((q ^ (c & 7)) << 4)) : "memory");
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int q = (sw & 1) * 4 + i;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int p = 32 * j + 4 * q + e;            // pixel = operand row
                            const unsigned at = dst + (unsigned)p * 128u + (unsigned)((((c >> 2) ^ (p & 7)) << 4) | ((c & 3) << 2));
                            asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(at), "r"(v[i][e] & TF32_MASK) : "memory");
                            asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(at + Y_STAGE), "r"(tf32_lo(v[i][e])) : "memory");
                        }
                    }
                    mbar_arrive(xempty0 + 8 * r);                                    // the ring slot can be refilled
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // generic writes -> tensor-core reads
                    mbar_arrive(ready0 + 8 * o);
                }
            }
        }
    } else {        // epilogue warps: warp w owns accumulator lanes 32w .. 32w+31 = pixels px0 + 32w + lane
        unsigned ti = 0;
        for (int tile = blockIdx.x; tile < a.total_tiles && ok; tile += gridDim.x, ++ti) {
            const unsigned buf = ti & 1u, tph = (ti >> 1) & 1u;
            TileAt at;
            const Problem &p = find_tile(a, tile, at);
            const int d = p.d, HW = p.HW, px = at.px0 + warp * 32 + lane;
            if (!mbar_wait_bounded(tfull0 + 8 * buf, tph)) { ok = false; break; }
            tc_fence_after();
            const unsigned taddr = tmem_base + ((unsigned)(warp * 32) << 16) + buf * acc_cols;
            const float *folded = p.bias != nullptr ? p.bias + (size_t)(p.w_per_image ? at.b : 0) * d : nullptr;
            const T *given = static_cast<const T *>(p.bias_as_given);
            TO *op = static_cast<TO *>(p.out) + (size_t)at.b * p.out_rows * HW + px;
            if (p.shuffle_w > 0) {
                const int y = px / p.shuffle_w, x = px - y * p.shuffle_w;
                op = static_cast<TO *>(p.out) + (size_t)at.b * p.out_rows * HW + (size_t)(4 * y) * p.shuffle_w + 2 * x;
            }
            for (int c0 = 0; c0 < d; c0 += 16) {
                unsigned r[16];
                tc_ld16(taddr + (unsigned)c0, r);
                tc_wait_ld();
                if (F32 && p.wide) {                    // second half of the accumulator: the x_hi * W'_lo term
                    unsigned r2[16];
                    tc_ld16(taddr + (unsigned)(d + c0), r2);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
                }
                if (c0 + 16 >= d) {                     // last read of this accumulator: hand it back to the MMA warp
                    tc_fence_before();
                    mbar_arrive(tempty0 + 8 * buf);
                }
                float v[16];
                if (folded != nullptr) {                // one branch for all: one per element costs more than the rest of the epilogue
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 t = load_current(reinterpret_cast<const float4 *>(folded + c0) + j);
                        v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
                    }
                } else if (!F32 && given != nullptr) {
                    if constexpr (!F32)
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const uint4 t = load_current(reinterpret_cast<const uint4 *>(given + c0) + j);
                            const unsigned w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float2 f = unpack_pair(T(), w[i]);
                                v[8 * j + 2 * i] = f.x; v[8 * j + 2 * i + 1] = f.y;
                            }
                        }
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = 0.f;
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
                if (px < HW && p.shuffle_w > 0) {
#pragma unroll
                    for (int j = 0; j < 16; j += 2) store_pair<TO>(op + (size_t)(c0 + (j & ~3)) * HW + (j & 2) * p.shuffle_w, v[j], v[j + 1]);
                } else if (px < HW) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) store_out(op + (size_t)(c0 + j) * HW, v[j]);
                }
            }
        }
    }
    if (!ok) atomicExch(&g_wait_timeout, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == MMA_WARP) tc_dealloc(tmem_base, (unsigned)a.tmem_cols);
}

// ---------------------------------------------------------------------------------- GroupNorm statistics and the fold
// one 16-byte load: 4 float32 or 8 16-bit elements, widened to float
template <typename T> struct Vec16 { static constexpr int N = 16 / (int)sizeof(T); };
__device__ __forceinline__ void load16(const float *p, float (&v)[4]) {
    const float4 t = __ldcs(reinterpret_cast<const float4 *>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void load16(const __half *p, float (&v)[8]) {
    const uint4 t = __ldcs(reinterpret_cast<const uint4 *>(p));
    const unsigned w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ void load16(const __nv_bfloat16 *p, float (&v)[8]) {
    const uint4 t = __ldcs(reinterpret_cast<const uint4 *>(p));
    const unsigned w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

__device__ __forceinline__ double block_sum(double v, double *scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    double t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += scratch[w];
    return t;       // valid in thread 0
}

struct StatProblem {
    const void *x;
    double2 *partial;               // [B * groups][nsplit]
    long long n;                    // (C / groups) * HW contiguous elements of a group
    int nsplit, blocks_end;         // blocks of the problems up to and including this one
};
struct StatList { StatProblem p[MAX_PROBLEMS]; int count; };

// block (s, bg) of a problem sums its slice of the n elements of group bg (16-byte loads, four in flight per thread; float
// partial sums of at most 32 elements, float64 beyond)
template <typename T>
__global__ void __launch_bounds__(STAT_THREADS) gn_partial_kernel(const __grid_constant__ StatList list) {
    begin_after_previous();
    constexpr int VN = Vec16<T>::N;
    __shared__ double scratch[STAT_THREADS / 32];
    int i = 0;
    while (i + 1 < list.count && (int)blockIdx.x >= list.p[i].blocks_end) ++i;
    const StatProblem &p = list.p[i];
    const int block = blockIdx.x - (i > 0 ? list.p[i - 1].blocks_end : 0), nsplit = p.nsplit, bg = block / nsplit;
    const T *base = static_cast<const T *>(p.x) + (size_t)bg * p.n;
    const long long vecs = p.n / VN, per = (vecs + nsplit - 1) / nsplit;
    const long long q0 = (block - bg * nsplit) * per, q1 = min(vecs, q0 + per);
    double s = 0, ss = 0;
    for (long long q = q0 + threadIdx.x; q < q1; q += 4 * STAT_THREADS) {
        float v[4][VN];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long qq = q + (long long)u * STAT_THREADS;
            if (qq < q1) {
                load16(base + qq * VN, v[u]);
            } else {
#pragma unroll
                for (int i = 0; i < VN; ++i) v[u][i] = 0.f;
            }
        }
        float fs = 0.f, fss = 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int i = 0; i < VN; ++i) { fs += v[u][i]; fss += v[u][i] * v[u][i]; }
        s += fs; ss += fss;
    }
    const double ts = block_sum(s, scratch), tss = block_sum(ss, scratch);
    if (threadIdx.x == 0) p.partial[block] = make_double2(ts, tss);
}

struct FoldProblem {
    const double2 *partial;         // nullptr: no norm
    const void *gamma, *beta, *weight, *bias;
    void *whi, *wlo;
    float *bias_out;
    long long n;
    int nsplit, C, groups, d, blocks_end;
    float eps;
};
struct FoldList { FoldProblem p[MAX_PROBLEMS]; int count; };

template <typename T> __device__ __forceinline__ void fetch16(const T *p, bool vec, float (&v)[Vec16<T>::N]) {
    if (vec) {
        load16(p, v);
    } else {
#pragma unroll
        for (int i = 0; i < Vec16<T>::N; ++i) v[i] = to_acc(load_current(p + i));
    }
}
// A block of a problem writes FOLD_ROWS rows of W'[b] (split in two for float32) and of bias'[b], a warp each.  The kernel is a chain
// of latencies: the statistics of the image (eight lanes share the slices of a group, the double division and root) and the loads of
// the parameters, which are under way meanwhile.  (A block per row, element by element: 7.0 us for the two projections of 16 images,
// d = 32, C = 256; this form 4.3.)
template <typename T>
__global__ void __launch_bounds__(STAT_THREADS) gn_fold_kernel(const __grid_constant__ FoldList list) {
    begin_after_previous();
    constexpr int VN = Vec16<T>::N;
    __shared__ float s_mean[MAX_GROUPS], s_rstd[MAX_GROUPS];
    int i = 0;
    while (i + 1 < list.count && (int)blockIdx.x >= list.p[i].blocks_end) ++i;
    const FoldProblem &p = list.p[i];
    const int block = blockIdx.x - (i > 0 ? list.p[i - 1].blocks_end : 0), d = p.d, per_image = (d + FOLD_ROWS - 1) / FOLD_ROWS, b = block / per_image,
              j = (block - b * per_image) * FOLD_ROWS + (threadIdx.x >> 5), lane = threadIdx.x & 31, groups = p.groups, C = p.C;
    const T *weight = static_cast<const T *>(p.weight) + (size_t)min(j, d - 1) * C, *bias = static_cast<const T *>(p.bias);
    const T *gamma = static_cast<const T *>(p.gamma), *beta = static_cast<const T *>(p.beta);
    const bool vec = ((reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta)) & 15u) == 0;
    float w[VN], ga[VN], be[VN];
    const auto fetch = [&](int c) {
        if (c >= C) return;               // rows are multiples of 16 bytes
        fetch16(weight + c, vec, w);
        if (groups > 0) { fetch16(gamma + c, vec, ga); fetch16(beta + c, vec, be); }
    };
    fetch(lane * VN);
    for (int g0 = 0; g0 < groups; g0 += STAT_THREADS / 8) {
        const int g = g0 + (threadIdx.x >> 3);
        double s = 0, ss = 0;
        if (g < groups)
            for (int k = threadIdx.x & 7; k < p.nsplit; k += 8) {
                const double2 t = p.partial[((size_t)b * groups + g) * p.nsplit + k];
                s += t.x; ss += t.y;
            }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        }
        if (g < groups && (threadIdx.x & 7) == 0) {
            const double mean = s / (double)p.n, var = fmax(ss / (double)p.n - mean * mean, 0.0);
            s_mean[g] = (float)mean;
            s_rstd[g] = (float)(1.0 / sqrt(var + (double)p.eps));
        }
    }
    __syncthreads();
    if (j >= d) return;
    const int cpg = groups > 0 ? C / groups : C;
    T *whi = static_cast<T *>(p.whi) + ((size_t)b * d + j) * C, *wlo = static_cast<T *>(p.wlo) + ((size_t)b * d + j) * C;
    double acc = 0;
    for (int c = lane * VN; c < C; c += 32 * VN) {
        float hi[VN], lo[VN];
        int g = c / cpg, next = (g + 1) * cpg - c;        // group of the element, elements up to the next group
#pragma unroll
        for (int e = 0; e < VN; ++e) {
            float scale = 1.f, shift = 0.f;
            if (e == next) { ++g; next += cpg; }
            if (groups > 0) {
                scale = ga[e] * s_rstd[g];
                shift = be[e] - s_mean[g] * scale;
            }
            const float wp = w[e] * scale;
            hi[e] = sizeof(T) == 4 ? __uint_as_float(__float_as_uint(wp) & TF32_MASK) : wp;
            lo[e] = wp - hi[e];
            acc += (double)w[e] * (double)shift;
        }
        if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4 *>(whi + c) = make_float4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<float4 *>(wlo + c) = make_float4(lo[0], lo[1], lo[2], lo[3]);
        } else {
            *reinterpret_cast<uint4 *>(whi + c) = make_uint4(pack_pair(T(), hi[0], hi[1]), pack_pair(T(), hi[2], hi[3]), pack_pair(T(), hi[4], hi[5]), pack_pair(T(), hi[6], hi[7]));
        }
        fetch(c + 32 * VN);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) p.bias_out[(size_t)b * d + j] = (float)(acc + (bias != nullptr ? (double)to_acc(bias[j]) : 0.0));
}

// ---------------------------------------------------------------------------------- host side
static size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }

// rows of one GEMM problem for d output rows: all of them up to 256, else equal parts of whole 16-row blocks
static int gemm_rows(int d) {
    for (int parts = 1; parts <= 4; ++parts)
        if (d % (16 * parts) == 0 && d / parts <= 256) return d / parts;
    return d;
}

// what the tensor-map / tcgen05 kernel takes: `rows` output rows in one problem
static bool problem_supported(int B, int C, int HW, int rows, int groups, int dtype) {
    if (dtype != SAPA_F32 && dtype != SAPA_F16 && dtype != SAPA_BF16) return false;
    const size_t esize = dtype_size(dtype);
    if (B <= 0 || C <= 0 || HW <= 0 || rows < 16 || rows > 256 || rows % 16 != 0) return false;
    if (((size_t)HW * esize) % 16 != 0 || ((size_t)C * esize) % 16 != 0) return false;     // tensor-map strides
    return groups >= 0 && groups <= MAX_GROUPS && (groups == 0 || (C % groups == 0 && ((size_t)(C / groups) * HW * esize) % 16 == 0));
}

// shared memory and tensor memory of a launch whose largest problem has `rows` output rows
struct Layout { int nx, no, acc_cols, tmem_cols; size_t smem; };
static bool is_wide(int rows, int esize) { return esize == 4 && 4 * rows <= 512; }      // two accumulators of 2 * rows columns must fit into TMEM
static bool make_layout(Layout &l, int rows, int acc_cols, int esize) {
    // operand slots: split activations + W' blocks (float32), W' block only (16-bit); the rest goes to the activation ring
    const size_t op = esize == 4 ? 2 * (size_t)Y_STAGE + 2 * (size_t)rows * 128 : (size_t)rows * 128;
    const size_t fixed = 1024 + 64 * 8;      // alignment slack + barriers
    l.no = esize == 4 ? OP_SLOTS_F32 : OP_SLOTS_16;
    if (fixed + l.no * op + 2 * (size_t)Y_STAGE > SMEM_LIMIT) return false;
    l.nx = (int)std::min<size_t>(MAX_SLOTS, (SMEM_LIMIT - fixed - l.no * op) / Y_STAGE);
    l.smem = fixed + l.no * op + (size_t)l.nx * Y_STAGE;
    l.acc_cols = acc_cols;
    l.tmem_cols = 32;
    while (l.tmem_cols < 2 * acc_cols) l.tmem_cols *= 2;
    return true;
}

// slices of a group for the statistics: as many as fill the eight blocks an SM holds on every SM, or, where that is more, of 32 KB, so that
// the last wave is a small part of the whole; at most MAX_SPLIT, which leaves a single group on 64 blocks and gives one of 16 MB slices of
// 256 KB
static int stat_splits(int B, int groups, long long n, int esize) {
    const long long fill = (148 * 8 + (long long)B * groups - 1) / ((long long)B * groups), even = (n * esize + STAT_SLICE - 1) / STAT_SLICE;
    return (int)std::max<long long>(1, std::min<long long>(MAX_SPLIT, std::max(fill, even)));
}

// One part (up to 256 rows) of a projection of the list, with the places of its intermediate results in the workspace.
struct Part {
    const sapa_projection *q;
    int rows, first_row, shuffle_w, nsplit;
    bool stats;                          // its statistics are taken for it (else an earlier part has them, or there are none)
    bool fold;                           // W' and bias' are written (else the weight is used as it is)
    size_t partial_ofs, whi_ofs, wlo_ofs, bias_ofs;
};
static bool same_norm(const sapa_projection &a, const sapa_projection &b) {
    return a.x == b.x && a.groups == b.groups && a.B == b.B && a.C == b.C && a.HW == b.HW;
}
// the parts of a list, and the bytes of workspace they need; 0: not supported.  With `list` false (the entry points for one projection,
// whose workspace query has sizes alone) everything is folded.
static size_t make_parts(Part *parts, int &count, const sapa_projection *p, const int *shuffle, int n, int dtype, bool list) {
    const int esize = (int)dtype_size(dtype);
    count = 0;
    size_t at = 0;
    for (int i = 0; i < n; ++i) {
        const sapa_projection &q = p[i];
        const int rows = q.d > 0 ? gemm_rows(q.d) : 0;
        Layout l;
        if (!problem_supported(q.B, q.C, q.HW, rows, q.groups, dtype) || !make_layout(l, rows, is_wide(rows, esize) ? 2 * rows : rows, esize)) return 0;
        for (int r = 0; r < q.d; r += rows) {
            Part &t = parts[count++];
            t.q = &q; t.rows = rows; t.first_row = r; t.shuffle_w = shuffle != nullptr ? shuffle[i] : 0;
            const int nimg = q.groups > 0 ? q.B : 1;
            t.nsplit = q.groups > 0 ? stat_splits(q.B, q.groups, (long long)(q.C / q.groups) * q.HW, esize) : 1;
            t.stats = q.groups > 0;
            t.fold = q.groups > 0 || esize == 4 || !list || !aligned16(q.bias) ||
                     !aligned16(static_cast<const unsigned char *>(q.weight) + (size_t)r * q.C * esize);
            for (int j = 0; j < count - 1 && t.stats; ++j)
                if (parts[j].stats && (parts[j].q == t.q || same_norm(*parts[j].q, q))) {
                    t.stats = false;
                    t.partial_ofs = parts[j].partial_ofs;
                }
            if (t.stats) { t.partial_ofs = at; at = round256(at + (size_t)q.B * q.groups * t.nsplit * sizeof(double2)); }
            if (t.fold) {
                t.whi_ofs = at; at = round256(at + (size_t)nimg * rows * q.C * esize);
                t.wlo_ofs = at; at = round256(at + (esize == 4 ? (size_t)nimg * rows * q.C * esize : 0));
                t.bias_ofs = at; at = round256(at + (size_t)nimg * rows * sizeof(float));
            }
        }
    }
    return std::max<size_t>(at, 256);
}

template <typename T, typename TO>
static int run_parts(const Part *parts, int count, unsigned char *ws, cudaStream_t st) {
    constexpr int KCH = 128 / (int)sizeof(T);
    constexpr CUtensorMapDataType type = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                         : std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    StatList sl{};
    FoldList fl{};
    int sblocks = 0, fblocks = 0;
    for (int i = 0; i < count; ++i) {
        const Part &t = parts[i];
        const sapa_projection &q = *t.q;
        if (t.stats) {
            StatProblem &s = sl.p[sl.count++];
            s.x = q.x; s.partial = reinterpret_cast<double2 *>(ws + t.partial_ofs); s.n = (long long)(q.C / q.groups) * q.HW; s.nsplit = t.nsplit;
            s.blocks_end = sblocks += q.B * q.groups * t.nsplit;
        }
        if (t.fold) {
            FoldProblem &f = fl.p[fl.count++];
            f.partial = q.groups > 0 ? reinterpret_cast<const double2 *>(ws + t.partial_ofs) : nullptr;
            f.gamma = q.gamma; f.beta = q.beta;
            f.weight = static_cast<const T *>(q.weight) + (size_t)t.first_row * q.C;
            f.bias = q.bias != nullptr ? static_cast<const T *>(q.bias) + t.first_row : nullptr;
            f.whi = ws + t.whi_ofs; f.wlo = ws + t.wlo_ofs; f.bias_out = reinterpret_cast<float *>(ws + t.bias_ofs);
            f.n = q.groups > 0 ? (long long)(q.C / q.groups) * q.HW : 1;
            f.nsplit = t.nsplit; f.C = q.C; f.groups = q.groups; f.d = t.rows; f.eps = q.eps;
            f.blocks_end = fblocks += ceil_div(t.rows, FOLD_ROWS) * (q.groups > 0 ? q.B : 1);
        }
    }
    if (sl.count > 0) {
        launch_next(gn_partial_kernel<T>, sblocks, STAT_THREADS, 0, st, sl);
        if (int e = check_launch("gn_partial_kernel")) return e;
    }
    if (fl.count > 0) {
        launch_next(gn_fold_kernel<T>, fblocks, STAT_THREADS, 0, st, fl);
        if (int e = check_launch("gn_fold_kernel")) return e;
    }

    Args a;
    a.count = count; a.total_tiles = 0; a.w_rows = 0;
    int acc_cols = 0;
    for (int i = 0; i < count; ++i) {      // the last input first: the statistics have just read it
        const Part &t = parts[count - 1 - i];
        const sapa_projection &q = *t.q;
        Problem &m = a.p[i];
        const int nimg = q.groups > 0 ? q.B : 1;
        const void *whi = t.fold ? ws + t.whi_ofs : static_cast<const void *>(static_cast<const T *>(q.weight) + (size_t)t.first_row * q.C);
        const void *wlo = t.fold && sizeof(T) == 4 ? ws + t.wlo_ofs : whi;
        if (!make_nchw_map(&m.x_map, q.x, q.HW, 1, q.C, q.B, KCH, KCH, 1, type, (int)sizeof(T), CU_TENSOR_MAP_SWIZZLE_128B) ||
            !make_nchw_map(&m.whi_map, whi, q.C, 1, t.rows, nimg, KCH, t.rows, 1, type, (int)sizeof(T), CU_TENSOR_MAP_SWIZZLE_128B) ||
            !make_nchw_map(&m.wlo_map, wlo, q.C, 1, t.rows, nimg, KCH, t.rows, 1, type, (int)sizeof(T), CU_TENSOR_MAP_SWIZZLE_128B)) {
            set_error("sapa_project_forward: tensor map creation failed (CUresult %d)", last_encode_result());
            return SAPA_ERR_UNSUPPORTED;
        }
        m.bias = t.fold ? reinterpret_cast<const float *>(ws + t.bias_ofs) : nullptr;
        m.bias_as_given = q.bias != nullptr ? static_cast<const T *>(q.bias) + t.first_row : nullptr;
        m.out = static_cast<TO *>(q.out) + (size_t)t.first_row * q.HW; m.out_rows = q.d; m.shuffle_w = t.shuffle_w;
        m.B = q.B; m.HW = q.HW; m.d = t.rows; m.w_per_image = q.groups > 0 ? 1 : 0;
        m.tiles_per_image = (q.HW + TILE_PX - 1) / TILE_PX;
        m.kblocks = (q.C + KCH - 1) / KCH;
        m.wide = is_wide(t.rows, (int)sizeof(T)) ? 1 : 0;
        m.tiles_end = a.total_tiles += m.tiles_per_image * q.B;
        a.w_rows = std::max(a.w_rows, t.rows);
        acc_cols = std::max(acc_cols, m.wide ? 2 * t.rows : t.rows);
    }
    Layout l;
    if (!make_layout(l, a.w_rows, acc_cols, (int)sizeof(T))) {
        set_error("sapa_project_forward: no layout for %d rows", a.w_rows);
        return SAPA_ERR_UNSUPPORTED;
    }
    a.nx = l.nx; a.no = l.no; a.tmem_cols = l.tmem_cols; a.acc_cols = acc_cols;
    int sms = 0;
    if (int e = prepare_launch(reinterpret_cast<const void *>(sapa_proj_umma_kernel<T, TO>), SMEM_LIMIT, "sapa_proj_umma_kernel", sms)) return e;
    launch_next(sapa_proj_umma_kernel<T, TO>, std::min(a.total_tiles, sms), THREADS, l.smem, st, a);
    return check_launch("sapa_proj_umma_kernel");
}

// the checked entry: `n` projections, in launches of up to MAX_PROBLEMS parts
static int run_list(const char *fn, const sapa_projection *p, const int *shuffle, int n, void *workspace, size_t workspace_bytes, int dtype, int out_dtype,
                    bool list, cudaStream_t st) {
    SAPA_REQUIRE(dtype_size(dtype) != 0, SAPA_ERR_DTYPE, "%s: unknown dtype code %d", fn, dtype);
    Part parts[MAX_LIST * 4];
    int count = 0;
    const bool types = out_dtype == dtype || (dtype == SAPA_F32 && (out_dtype == SAPA_F16 || out_dtype == SAPA_BF16));
    const size_t need = p != nullptr && n >= 1 && n <= MAX_LIST && types ? make_parts(parts, count, p, shuffle, n, dtype, list) : 0;
    SAPA_REQUIRE(need != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: needs float32 / float16 / bfloat16 (output of the same type, or 16 bits of float32), d a multiple of 16 up to 1024, rows of HW and C "
                 "elements that are multiples of 16 bytes and C divisible by groups", fn);
    for (int i = 0; i < n; ++i) {
        const void *x = p[i].x, *gamma = p[i].gamma, *beta = p[i].beta, *weight = p[i].weight, *out = p[i].out;
        SAPA_CHECK_PTR(fn, x); SAPA_CHECK_PTR(fn, weight);
        if (p[i].groups > 0) { SAPA_CHECK_PTR(fn, gamma); SAPA_CHECK_PTR(fn, beta); }
        SAPA_REQUIRE(out != nullptr && all_aligned16(x, out), SAPA_ERR_ALIGNMENT, "%s: x and out must be 16-byte aligned", fn);
    }
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 256 == 0, SAPA_ERR_WORKSPACE,
                 "%s: a 256-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    for (int i = 0; i < n && shuffle != nullptr; ++i)
        SAPA_REQUIRE(shuffle[i] >= 0 && (shuffle[i] == 0 || p[i].HW % shuffle[i] == 0), SAPA_ERR_ARGUMENT, "%s: bad shuffle width", fn);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    for (int i = 0; i < count; i += MAX_PROBLEMS) {
        const int m = std::min(MAX_PROBLEMS, count - i);
        int e;
        if (dtype == SAPA_F16) e = run_parts<__half, __half>(parts + i, m, ws, st);
        else if (dtype == SAPA_BF16) e = run_parts<__nv_bfloat16, __nv_bfloat16>(parts + i, m, ws, st);
        else if (out_dtype == SAPA_F16) e = run_parts<float, __half>(parts + i, m, ws, st);
        else if (out_dtype == SAPA_BF16) e = run_parts<float, __nv_bfloat16>(parts + i, m, ws, st);
        else e = run_parts<float, float>(parts + i, m, ws, st);
        if (e) return e;
    }
    return SAPA_OK;
}

// workspace of one projection of which only the sizes are known
static size_t one_workspace(int B, int C, int HW, int d, int groups, int dtype) {
    sapa_projection q{};
    q.B = B; q.C = C; q.HW = HW; q.d = d; q.groups = groups;
    Part parts[4];
    int count = 0;
    return make_parts(parts, count, &q, nullptr, 1, dtype, false);
}

}  // namespace proj

int proj_wait_timeout_flag() {
    int flag = 0;
    if (cudaMemcpyFromSymbol(&flag, proj::g_wait_timeout, sizeof(int)) != cudaSuccess) return -1;
    if (flag != 0) {
        const int zero = 0;
        if (cudaMemcpyToSymbol(proj::g_wait_timeout, &zero, sizeof(int)) != cudaSuccess) return -1;
    }
    return flag;
}

}  // namespace sapa

using namespace sapa;

extern "C" {

size_t sapa_project_workspace(int B, int C, int HW, int d, int groups, int dtype) {
    return d <= 256 ? proj::one_workspace(B, C, HW, d, groups, dtype) : 0;
}

int sapa_project_forward(const void *x, const void *gamma, const void *beta, const void *weight, const void *bias, void *out,
                         void *workspace, size_t workspace_bytes, int B, int C, int HW, int d, int groups, float eps, int dtype,
                         void *stream) {
    const char *fn = "sapa_project_forward";
    trace_reset();
    SAPA_REQUIRE(dtype_size(dtype) != 0, SAPA_ERR_DTYPE, "%s: unknown dtype code %d", fn, dtype);
    SAPA_REQUIRE(sapa_project_workspace(B, C, HW, d, groups, dtype) != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: needs float32 / float16 / bfloat16, d a multiple of 16 up to 256, rows of HW and C elements that are "
                 "multiples of 16 bytes and C divisible by groups (got B=%d C=%d HW=%d d=%d groups=%d)", fn, B, C, HW, d, groups);
    SAPA_CHECK_PTR(fn, x); SAPA_CHECK_PTR(fn, weight); SAPA_CHECK_PTR(fn, out);
    const sapa_projection q{x, gamma, beta, weight, bias, out, nullptr, B, C, HW, d, groups, eps};
    return proj::run_list(fn, &q, nullptr, 1, workspace, workspace_bytes, dtype, dtype, false, static_cast<cudaStream_t>(stream));
}

size_t sapa_project_rows_workspace(int B, int C, int HW, int d, int groups, int dtype) { return proj::one_workspace(B, C, HW, d, groups, dtype); }

int sapa_project_rows_forward(const void *x, const void *gamma, const void *beta, const void *weight, const void *bias, void *out, int shuffle_width,
                              void *workspace, size_t workspace_bytes, int B, int C, int HW, int d, int groups, float eps, int dtype, int out_dtype,
                              void *stream) {
    trace_reset();
    const sapa_projection q{x, gamma, beta, weight, bias, out, nullptr, B, C, HW, d, groups, eps};
    return proj::run_list("sapa_project_rows_forward", &q, &shuffle_width, 1, workspace, workspace_bytes, dtype, out_dtype, false, static_cast<cudaStream_t>(stream));
}

size_t sapa_project_list_workspace(const sapa_projection *p, int count, int dtype) {
    proj::Part parts[proj::MAX_LIST * 4];
    int n = 0;
    if (p == nullptr || count < 1 || count > proj::MAX_LIST) return 0;
    for (int i = 0; i < count; ++i)
        if (p[i].d <= 0 || p[i].d > 1024) return 0;
    return proj::make_parts(parts, n, p, nullptr, count, dtype, true);
}

int sapa_project_list_forward(const sapa_projection *p, const int *shuffle_widths, int count, void *workspace, size_t workspace_bytes, int dtype,
                              int out_dtype, void *stream) {
    trace_reset();
    return proj::run_list("sapa_project_list_forward", p, shuffle_widths, count, workspace, workspace_bytes, dtype, out_dtype, true, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
