// sapa_strip_sim.cuh — the float32 logits  S_k(p) = sum_c X_c(p) L_c(win_k(p))  (K = 5, s = 2) on the 5th-generation tensor cores, and what
// follows them per pixel: nothing (the similarity by itself), the softmax (first half of the forward), or the softmax backward with the
// saved attention map (stage 1 of the backward).  The aggregation that comes next is sapa_strip.cuh's.  Included by sapa_tma.cu.
//
// A unit is two low-res rows of a strip of 16 columns: its four high-res rows of 32 pixels are the 128 lanes of ONE product
//     S[128 px x 120 cells] += X^T[128 px x 32 ch] * L[32 ch x 120 cells],       cells = six rows of the 20 columns that the windows reach
// per 32 channels, three terms of tf32, the small products of a stage first.  An accumulation in tensor memory rounds toward zero, twelve times a
// stage, which numbers of one sign feel most: a product is of 64 channels at most, and the sums of those are added in registers (features of one sign,
// logits of 256 channels 4.7e-6 from float64 in one product, 9.6e-7 in four, of 720 1.6e-5 and 9.5e-7; on tiles 5.2e-6, 1.6e-5; times the same).
//   * X: a warpgroup reads the landed box (lane = pixel, a channel at a time) and writes both terms to tensor memory as the A operand.
//   * L: eight warps turn the landed box into rows of channels (unswizzled 8 x 16 byte core matrices) and split it.
//   * per pixel: a thread reads the 20 cells that its row of pixels reaches of each of its five window rows, shifts its own five to the
//     front and holds its 25 logits: no shuffles.  Two warpgroups take turns.
namespace ssim {

using namespace ummau;

constexpr int CELLS = 16, SPAN = 20, ROWS6 = 6, N = 128;    // columns of a strip; cells of a row, rows; operand rows (120, rounded up)
constexpr int KCH = 32, PART = 2;                           // channels of a stage, stages of a product
constexpr int PIX_WARPS = 8, X_WARP0 = 8, L_WARP0 = 12, L_WARPS = 8, TMA_WARP = 20, MMA_WARP = 21, NT = 22 * 32;
constexpr int LROW = 112, X_BYTES = 4 * KCH * 128, L_BYTES = ROWS6 * KCH * LROW, SLOT = X_BYTES + L_BYTES, NL = 4;
constexpr int B_LBO = N * 16, B_TERM = KCH / 4 * B_LBO, B_BYTES = 2 * B_TERM, NB = 2;              // a buffer for each of the two warpgroups that write L
constexpr int NA = 4, A_COL = 2 * N, TMEM_COLS = 512;       // accumulators at 0 and N; A operands of 64 columns
constexpr int SMEM = NL * SLOT + NB * B_BYTES + 1024;
static_assert(SMEM <= 227 * 1024 && A_COL + NA * 2 * KCH <= TMEM_COLS && SLOT % 128 == 0, "layout");
constexpr int LOGITS = 0, SOFTMAX = 1, SOFTMAX_BWD = 2;

struct Args {
    const float *attn;     // SOFTMAX_BWD: the saved map
    float *out;            // [B, 25, 2 map_rows, 2W], from low-res row map_y0 on: logits, attention map or logit gradients
    int map_rows, map_y0;
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
}  // namespace ssim

template <int WHAT>
__global__ void __launch_bounds__(ssim::NT, 1) sapa_strip_sim_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap lmap, const ssim::Args a) {
    using namespace ummau;
    namespace Z = ssim;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * (Z::NL + Z::NA + Z::NB) + 6];
    __shared__ unsigned tmem_slot;
    const unsigned ring = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u, bop = ring + Z::NL * Z::SLOT;
    const unsigned full = (unsigned)__cvta_generic_to_shared(bars), empty = full + 8 * Z::NL, aready = empty + 8 * Z::NL, aempty = aready + 8 * Z::NA;
    const unsigned bready = aempty + 8 * Z::NA, bempty = bready + 8 * Z::NB, sfull = bempty + 8 * Z::NB, sempty = sfull + 32;      // sfull: [warpgroup that takes the unit][accumulator]
    const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
    const int units = a.B * a.pairs * a.strips;

    if (tid == 0) {
        for (int i = 0; i < Z::NL; ++i) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, 128 + 128); }
        for (int i = 0; i < Z::NA; ++i) { mbar_init(aready + 8 * i, 128); mbar_init(aempty + 8 * i, 1); }
        for (int i = 0; i < Z::NB; ++i) { mbar_init(bready + 8 * i, 128); mbar_init(bempty + 8 * i, 1); }
        for (int i = 0; i < 4; ++i) mbar_init(sfull + 8 * i, 1);
        for (int i = 0; i < 2; ++i) mbar_init(sempty + 8 * i, 128);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == Z::MMA_WARP) {
        tc_alloc((unsigned)__cvta_generic_to_shared(&tmem_slot), Z::TMEM_COLS);
        tc_relinquish();
    }
    for (int i = tid; i < Z::NB * Z::B_BYTES / 16; i += Z::NT)        // the operand rows beyond the cells stay zero
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(bop + 16 * i), "r"(0u) : "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = warp_uniform(*reinterpret_cast<volatile unsigned *>(&tmem_slot));
    const unsigned quarter = (unsigned)((warp & 3) * 32) << 16;       // the lanes of tensor memory that a warp can reach
    begin_after_previous();

    bool ok = true;
    if (warp == Z::TMA_WARP) {
        if (lane == 0) {
            int slot = 0, phase = 0;
            for (int i = blockIdx.x; i < units && ok; i += gridDim.x) {
                const Z::Unit u = Z::unit_at(a, i);
                for (int s = 0; s < a.stages; ++s) {
                    if (!mbar_wait_bounded(empty + 8 * slot, phase ^ 1)) { ok = false; break; }
                    mbar_expect_tx(full + 8 * slot, Z::SLOT);
                    tma_load_4d(ring + slot * Z::SLOT, &xmap, full + 8 * slot, 2 * u.x0, s * Z::KCH, 2 * u.y, u.n);
                    tma_load_4d(ring + slot * Z::SLOT + Z::X_BYTES, &lmap, full + 8 * slot, u.x0 - 4, s * Z::KCH, a.ytop0 + u.y - 2, u.n);
                    if (++slot == Z::NL) { slot = 0; phase ^= 1; }
                }
            }
            if (!ok) (void)drain_loads<Z::NL>(full, slot, phase);     // none of its loads may land after it has left
        }
    } else if (warp == Z::MMA_WARP) {
        constexpr unsigned HI = (128u >> 4) | (1u << 14), IDESC = IDESC_M128<float> | idesc_n(Z::N);
        const unsigned leader = elect_leader(), b_base = warp_uniform(desc_lo(bop, Z::B_LBO));
        int ab = 0, aph = 0, bb = 0, bph = 0, part = 0, group = 0;
        for (int i = blockIdx.x; i < units && ok; i += gridDim.x, group ^= 1)
            for (int s = 0; s < a.stages && ok; ++s) {
                const int buf = part & 1, in = s % Z::PART;           // stage of its product
                if (in == 0) ok = mbar_wait_warp(sempty + 8 * buf, ((part >> 1) & 1) ^ 1);
                ok = ok && mbar_wait_warp(aready + 8 * ab, aph) && mbar_wait_warp(bready + 8 * bb, bph);
                if (!ok) break;
                const unsigned d = tmem + buf * Z::N;
                tc_fence_after();
                const unsigned at = tmem + Z::A_COL + ab * 2 * Z::KCH, b = b_base + ((bb * Z::B_BYTES) >> 4);
                constexpr unsigned KB = 2 * Z::B_LBO >> 4;            // 8 channels further
                auto product = [&](auto steps) {
                    constexpr int KS = decltype(steps)::value;
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) tc_mma_ta<true>(leader, d, at + Z::KCH + 8 * ks, b + ks * KB, HI, IDESC, in > 0 || ks > 0 ? 1u : 0u);
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) tc_mma_ta<true>(leader, d, at + 8 * ks, b + (Z::B_TERM >> 4) + ks * KB, HI, IDESC, 1u);
#pragma unroll
                    for (int ks = 0; ks < KS; ++ks) tc_mma_ta<true>(leader, d, at + 8 * ks, b + ks * KB, HI, IDESC, 1u);
                };
                if (a.d - s * Z::KCH > 16) product(std::integral_constant<int, 4>{});
                else product(std::integral_constant<int, 2>{});       // the channels end in the first half of the stage
                tc_commit_by(leader, aempty + 8 * ab);
                tc_commit_by(leader, bempty + 8 * bb);
                if (++ab == Z::NA) { ab = 0; aph ^= 1; }
                if (++bb == Z::NB) { bb = 0; bph ^= 1; }
                if (in == Z::PART - 1 || s == a.stages - 1) {
                    tc_commit_by(leader, sfull + 16 * group + 8 * buf);
                    ++part;
                }
            }
    } else if (warp >= Z::X_WARP0 && warp < Z::L_WARP0) {
        int slot = 0, phase = 0, ab = 0, aph = 0;
        for (int i = blockIdx.x; i < units && ok; i += gridDim.x)
            for (int s = 0; s < a.stages; ++s) {
                if (!mbar_wait_warp(full + 8 * slot, phase) || !mbar_wait_warp(aempty + 8 * ab, aph ^ 1)) { ok = false; break; }
                tc_fence_after();
                const unsigned src = fresh(ring + slot * Z::SLOT + (warp & 3) * (Z::KCH * 128) + lane * 4), at = tmem + quarter + Z::A_COL + ab * 2 * Z::KCH;
#pragma unroll
                for (int h = 0; h < Z::KCH / 16; ++h) {
                    if (16 * h >= a.d - s * Z::KCH) break;
                    unsigned v[16];
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] = lds32(src + (16 * h + c) * 128);
                    tc_st16(at + 16 * h, v);                          // the tensor core reads the top 19 bits of a tf32 operand
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] = tf32_lo(v[c]);
                    tc_st16(at + Z::KCH + 16 * h, v);
                }
                mbar_arrive(empty + 8 * slot);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(aready + 8 * ab);
                if (++slot == Z::NL) { slot = 0; phase ^= 1; }
                if (++ab == Z::NA) { ab = 0; aph ^= 1; }
            }
    } else if (warp >= Z::L_WARP0 && warp < Z::TMA_WARP) {
        // a thread writes operand row (cell) n, four channels at a time; a warpgroup for each operand buffer: every second stage
        const int group = (warp - Z::L_WARP0) >> 2, n = (warp & 3) * 32 + lane;
        const bool live = n < Z::ROWS6 * Z::SPAN;
        const unsigned from = Z::X_BYTES + (live ? n / Z::SPAN * (Z::KCH * Z::LROW) + (n % Z::SPAN + 2) * 4 : 0), to = (n >> 3) * 128 + (n & 7) * 16;
        int slot = 0, phase = 0, bph = 0, stage = 0;
        for (int i = blockIdx.x; i < units && ok; i += gridDim.x)
            for (int s = 0; s < a.stages; ++s, ++stage) {
                if ((stage & 1) == group) {
                    if (!mbar_wait_bounded(full + 8 * slot, phase) || !mbar_wait_bounded(bempty + 8 * group, bph ^ 1)) { ok = false; break; }
                    bph ^= 1;
                    const unsigned src = fresh(ring + slot * Z::SLOT + from), dst = bop + group * Z::B_BYTES + to;
                    if (live)
#pragma unroll
                        for (int q = 0; q < Z::KCH / 4; ++q) {
                            if (4 * q >= a.d - s * Z::KCH && (q & 3) == 0) break;         // only half of the stage is read
                            unsigned v[4];
#pragma unroll
                            for (int c = 0; c < 4; ++c) v[c] = lds32(src + (4 * q + c) * Z::LROW);
                            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(dst + q * Z::B_LBO), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
                            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(dst + Z::B_TERM + q * Z::B_LBO), "r"(tf32_lo(v[0])), "r"(tf32_lo(v[1])),
                                         "r"(tf32_lo(v[2])), "r"(tf32_lo(v[3])) : "memory");
                        }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    mbar_arrive(bready + 8 * group);
                    mbar_arrive(empty + 8 * slot);
                }
                if (++slot == Z::NL) { slot = 0; phase ^= 1; }
            }
    } else if (warp < Z::PIX_WARPS) {
        // thread = lane of S: pixel `lane` of high-res row (warp & 3) of the unit, whose low-res row is (warp & 3) / 2
        const int group = warp >> 2, row = warp & 3, shift = lane >> 1;
        const unsigned from0 = tmem + quarter + (row >> 1) * Z::SPAN;
        const int parts = (a.stages + Z::PART - 1) / Z::PART;
        const size_t hi_plane = (size_t)(2 * a.map_rows) * (2 * a.W);
        int step = 0, ph = 0;                                         // bit b of ph: the phase of accumulator b
        for (int i = blockIdx.x; i < units && ok; i += gridDim.x, ++step) {
            if ((step & 1) != group) continue;
            const Z::Unit u = Z::unit_at(a, i);
            const bool inside = u.y + (row >> 1) < a.y_end && u.x0 + shift < a.W;
            const size_t at = (size_t)u.n * 25 * hi_plane + (size_t)(2 * (u.y - a.map_y0) + row) * (2 * a.W) + 2 * u.x0 + lane;
            float w[WHAT == Z::SOFTMAX_BWD ? 25 : 1];
            if (WHAT == Z::SOFTMAX_BWD)
#pragma unroll
                for (int k = 0; k < 25; ++k) w[WHAT == Z::SOFTMAX_BWD ? k : 0] = inside ? a.attn[at + k * hi_plane] : 0.f;
            float s[25];
            for (int p = 0; p < parts; ++p) {
                const int buf = (step * parts + p) & 1;
                const unsigned from = from0 + buf * Z::N;
                if (!mbar_wait_warp(sfull + 16 * group + 8 * buf, ph >> buf & 1)) { ok = false; break; }
                ph ^= 1 << buf;
                tc_fence_after();
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) {
                    unsigned t[20];
                    tc_ld16(from + dy * Z::SPAN, *reinterpret_cast<unsigned (*)[16]>(&t[0]));
                    sfwd::tc_ld4(from + dy * Z::SPAN + 16, &t[16]);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 12; ++e) t[e] = shift & 8 ? t[e + 8] : t[e];
#pragma unroll
                    for (int e = 0; e < 8; ++e) t[e] = shift & 4 ? t[e + 4] : t[e];
#pragma unroll
                    for (int e = 0; e < 6; ++e) t[e] = shift & 2 ? t[e + 2] : t[e];
#pragma unroll
                    for (int e = 0; e < 5; ++e) {
                        const float x = __uint_as_float(shift & 1 ? t[e + 1] : t[e]);
                        s[5 * dy + e] = p > 0 ? s[5 * dy + e] + x : x;
                    }
                }
                tc_fence_before();
                mbar_arrive(sempty + 8 * buf);
            }
            if (!ok) break;
            if (WHAT == Z::SOFTMAX) {
                float m = s[0], z = 0.f;
#pragma unroll
                for (int k = 1; k < 25; ++k) m = fmaxf(m, s[k]);
#pragma unroll
                for (int k = 0; k < 25; ++k) s[k] = expf(s[k] - m);
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) z += ((s[5 * dy] + s[5 * dy + 1]) + (s[5 * dy + 2] + s[5 * dy + 3])) + s[5 * dy + 4];
                const float inv = 1.f / z;
#pragma unroll
                for (int k = 0; k < 25; ++k) s[k] *= inv;
            }
            if (WHAT == Z::SOFTMAX_BWD) {
                float dot = 0.f;
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) {
                    float part = 0.f;
#pragma unroll
                    for (int e = 0; e < 5; ++e) part = fmaf(w[WHAT == Z::SOFTMAX_BWD ? 5 * dy + e : 0], s[5 * dy + e], part);
                    dot += part;
                }
#pragma unroll
                for (int k = 0; k < 25; ++k) s[k] = w[WHAT == Z::SOFTMAX_BWD ? k : 0] * (s[k] - dot);
            }
            if (inside)
#pragma unroll
                for (int k = 0; k < 25; ++k) a.out[at + k * hi_plane] = s[k];
        }
    }
    if (!ok) atomicExch(&g_wait_timeout, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == Z::MMA_WARP) tc_dealloc(tmem, Z::TMEM_COLS);
}
