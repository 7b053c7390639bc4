// sapa_strip_sim16.cuh — sapa_strip_sim.cuh in 16 bits: the logits of two low-res rows of a strip of 32 columns, and per pixel nothing (the
// similarity by itself, in 16 bits or as float32) or the softmax backward with the saved attention map (stage 1 of the backward; the
// aggregation that comes next is sapa_strip.cuh's).  Included by sapa_tma.cu.
//
// A low-res row is a tile: its two high-res rows of 64 pixels are the 128 lanes of
//     S[128 px x 48 cells] += X^T[128 px x KCH ch] * L[KCH ch x 48 cells]         per window row;
// the two tiles of a unit share six rows of L.  Both operands are what TMA lands (channel rows of 128 bytes: "MN-major", 128-byte
// swizzle), so there is nothing to do but to load, to issue and to finish the pixels: a warpgroup for each tile, thread = pixel, whose
// five cells of a row are shifted to the front (sapa_strip_fwd.cuh).  What bounds it: with many channels the MMAs' reads of shared
// memory (each reads the 128 pixels again: 44 clocks measured instead of 24; 256 channels under ncu: tensor pipe 36 %, memory 40 % of the time), with few
// the pixels and their 25 values.
namespace s16 {

using namespace ummau;

constexpr int CELLS = 32, SN = 48, ROWS6 = 6;               // columns of a strip, cells of a row of logits (columns x0 - 8 and so on), rows of L
constexpr int PIX_WARPS = 8, TMA_WARP = 8, MMA_WARP = 9, NT = 10 * 32;
constexpr int TILE_COLS = 5 * SN, TMEM_COLS = 512;
constexpr int MAX_NL = 10;
constexpr int LOGITS = 0, LOGITS_F32 = 1, SOFTMAX_BWD = 2;

template <int KCH> struct Lay {
    static constexpr int ROW = KCH * 128, X_BYTES = 4 * ROW, L_BYTES = ROWS6 * ROW, SLOT = X_BYTES + L_BYTES, NL = KCH == 16 ? 10 : 5;
    static constexpr int SMEM = NL * SLOT + 1024;
    static_assert(SMEM <= 227 * 1024 && NL <= MAX_NL && ROW % 1024 == 0 && 2 * TILE_COLS <= TMEM_COLS, "layout");
};
struct Args {
    const void *attn;      // SOFTMAX_BWD: the saved map
    void *out;             // [B, 25, 2H, 2W]: logits or logit gradients
    int B, d, H, W, ytop0, y_begin, y_end;
    int strips, pairs, stages;
};
struct Unit { int n, x0, y; };
__device__ __forceinline__ Unit unit_at(const Args &a, int i) {
    Unit u;
    u.x0 = (i % a.strips) * CELLS; i /= a.strips;
    u.y = a.y_begin + 2 * (i % a.pairs);
    u.n = i / a.pairs;
    return u;
}
}  // namespace s16

template <typename T, int WHAT, int KCH>
__global__ void __launch_bounds__(s16::NT, 1) sapa_strip_sim_16_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap lmap,
                                                                       const s16::Args a) {
    using namespace ummau;
    namespace Z = s16;
    using L = Z::Lay<KCH>;
    using O = typename std::conditional<WHAT == Z::LOGITS_F32, float, T>::type;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * (Z::MAX_NL + 2)];
    __shared__ unsigned tmem_slot;
    const unsigned ring = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned full = (unsigned)__cvta_generic_to_shared(bars), empty = full + 8 * Z::MAX_NL, sfull = empty + 8 * Z::MAX_NL, sempty = sfull + 16;
    const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
    const int units = a.B * a.pairs * a.strips;

    if (tid == 0) {
        for (int i = 0; i < L::NL; ++i) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(sfull + 8 * i, 1); mbar_init(sempty + 8 * i, 128); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == Z::MMA_WARP) {
        tc_alloc((unsigned)__cvta_generic_to_shared(&tmem_slot), Z::TMEM_COLS);
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = warp_uniform(*reinterpret_cast<volatile unsigned *>(&tmem_slot));
    begin_after_previous();

    bool ok = true;
    if (warp == Z::TMA_WARP) {
        if (lane == 0) {
            int slot = 0, phase = 0;
            for (int i = blockIdx.x; i < units && ok; i += gridDim.x) {
                const Z::Unit u = Z::unit_at(a, i);
                for (int s = 0; s < a.stages; ++s) {
                    if (!mbar_wait_bounded(empty + 8 * slot, phase ^ 1)) { ok = false; break; }
                    mbar_expect_tx(full + 8 * slot, L::SLOT);
                    tma_load_4d(ring + slot * L::SLOT, &xmap, full + 8 * slot, 2 * u.x0, s * KCH, 2 * u.y, u.n);
                    tma_load_4d(ring + slot * L::SLOT + L::X_BYTES, &lmap, full + 8 * slot, u.x0 - 8, s * KCH, a.ytop0 + u.y - 2, u.n);
                    if (++slot == L::NL) { slot = 0; phase ^= 1; }
                }
            }
            if (!ok) (void)drain_loads<L::NL>(full, slot, phase);     // none of its loads may land after it has left
        }
    } else if (warp == Z::MMA_WARP) {
        constexpr unsigned HI = (1024u >> 4) | (1u << 14) | (2u << 29);         // 8 channels of 128 bytes, 128-byte swizzle
        constexpr unsigned IDESC = IDESC_M128<T> | (1u << 15) | (1u << 16) | idesc_n(Z::SN);       // both operands MN-major
        const unsigned leader = elect_leader(), x_base = warp_uniform(desc_lo(ring, L::ROW));
        int slot = 0, phase = 0, par = 1;
        for (int i = blockIdx.x; i < units && ok; i += gridDim.x, par ^= 1)
            for (int s = 0; s < a.stages && ok; ++s) {
                ok = mbar_wait_warp(full + 8 * slot, phase);
                const unsigned x = x_base + ((slot * L::SLOT) >> 4), l = x + (L::X_BYTES >> 4);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (s == 0) ok = ok && mbar_wait_warp(sempty + 8 * t, par);           // the unit before has been read
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                        for (int ks = 0; ks < KCH / 16; ++ks)
                            tc_mma<false>(leader, tmem + t * Z::TILE_COLS + dy * Z::SN, x + ((2 * t * L::ROW + ks * 2048) >> 4),
                                          l + (((t + dy) * L::ROW + ks * 2048) >> 4), HI, IDESC, s > 0 || ks > 0 ? 1u : 0u);
                    if (s == a.stages - 1) tc_commit_by(leader, sfull + 8 * t);
                }
                if (!ok) break;
                tc_commit_by(leader, empty + 8 * slot);
                if (++slot == L::NL) { slot = 0; phase ^= 1; }
            }
    } else {
        // thread = lane of S: pixel px of high-res row r of its warpgroup's tile
        const int tile = warp >> 2, r = (warp >> 1) & 1, px = (warp & 1) * 32 + lane, shift = lane >> 1;
        const unsigned from = tmem + ((unsigned)((warp & 3) * 32) << 16) + tile * Z::TILE_COLS + (warp & 1) * 16 + 6;
        const size_t hi_plane = (size_t)(2 * a.H) * (2 * a.W);
        int ph = 0;
        for (int i = blockIdx.x; i < units; i += gridDim.x, ph ^= 1) {
            const Z::Unit u = Z::unit_at(a, i);
            const int y = u.y + tile;
            const bool inside = y < a.y_end && u.x0 + (px >> 1) < a.W;
            const size_t at = (size_t)u.n * 25 * hi_plane + (size_t)(2 * y + r) * (2 * a.W) + 2 * u.x0 + px;
            T w[WHAT == Z::SOFTMAX_BWD ? 25 : 1];
            if (WHAT == Z::SOFTMAX_BWD)
#pragma unroll
                for (int k = 0; k < 25; ++k) w[WHAT == Z::SOFTMAX_BWD ? k : 0] = inside ? static_cast<const T *>(a.attn)[at + k * hi_plane] : from_acc<T>(0.f);
            if (!mbar_wait_warp(sfull + 8 * tile, ph)) { ok = false; break; }
            tc_fence_after();
            float s[25];
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {
                unsigned t[20];
                tc_ld16(from + dy * Z::SN, *reinterpret_cast<unsigned (*)[16]>(&t[0]));
                sfwd::tc_ld4(from + dy * Z::SN + 16, &t[16]);
                tc_wait_ld();
#pragma unroll
                for (int e = 0; e < 12; ++e) t[e] = shift & 8 ? t[e + 8] : t[e];
#pragma unroll
                for (int e = 0; e < 8; ++e) t[e] = shift & 4 ? t[e + 4] : t[e];
#pragma unroll
                for (int e = 0; e < 6; ++e) t[e] = shift & 2 ? t[e + 2] : t[e];
#pragma unroll
                for (int e = 0; e < 5; ++e) s[5 * dy + e] = __uint_as_float(shift & 1 ? t[e + 1] : t[e]);
            }
            tc_fence_before();
            mbar_arrive(sempty + 8 * tile);
            if (WHAT == Z::SOFTMAX_BWD) {
                float dot = 0.f;
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) {
                    float part = 0.f;
#pragma unroll
                    for (int e = 0; e < 5; ++e) part = fmaf(to_acc(w[WHAT == Z::SOFTMAX_BWD ? 5 * dy + e : 0]), s[5 * dy + e], part);
                    dot += part;
                }
#pragma unroll
                for (int k = 0; k < 25; ++k) s[k] = to_acc(w[WHAT == Z::SOFTMAX_BWD ? k : 0]) * (s[k] - dot);
            }
            if (inside)
#pragma unroll
                for (int k = 0; k < 25; ++k) static_cast<O *>(a.out)[at + k * hi_plane] = from_acc<O>(s[k]);
        }
    }
    if (!ok) atomicExch(&g_wait_timeout, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == Z::MMA_WARP) tc_dealloc(tmem, Z::TMEM_COLS);
}
