// sapa_tma.cu — SAPA-B for K = 5, s = 2 with TMA staging and the contractions on the tensor cores: one float32 kernel
// and one float16 / bfloat16 kernel on tiles, each in four modes (fused forward, stage 1 of the fused backward, logits only,
// aggregation only), and the choice between them and the kernels on strips of columns (tcgen05, sapa_strip*.cuh), which take the larger
// problems with rows of 16 bytes.
//
// Same mathematics as sapa_mma.cu (probabilities kept in registers between the logit MMAs and the aggregation
// MMAs), but the key / query / value tiles are brought into shared memory by the tensor memory accelerator instead
// of per-lane cp.async copies.  Measured reason: with 64-byte row segments the cp.async path delivers about one
// 16-byte lane-copy per clock per SM (4.6 TB/s over the GPU), which alone costs 43 us at B=8, C=256, d=64,
// 64x64 -> 128x128, more than the HBM time of the whole op.  One elected thread issues one cp.async.bulk.tensor per tile:
//   * tensors are described as 4-D maps (x, channel, y, image); a box of BW columns x NCH channels x 8 rows lands
//     in shared memory as [row][channel][BW columns] (float32: 16 columns = 64-byte rows with the 64-byte swizzle);
//   * coordinates outside the tensor (image border, tile overhang, channel tails) are filled with zeros by the
//     hardware, which is exactly the reference's border rule;
//   * completion is signalled on an mbarrier per ring slot (expect_tx = box bytes); every wait is bounded and
//     raises a device-side error flag instead of spinning for ever.
// With channel-minor rows of 64 bytes and the 64-byte swizzle, the per-lane fragment loads of the float32
// aggregation (lane = 4 * channel + cell) touch 32 different banks.
//
// float32 computes the logits on the tensor cores as well (3 x tf32, M = 16 pixels, N = 8 window cells, K = 8
// channels): on the FP32 pipe that loop was bound by shared-memory wavefronts (12 per 10 packed FMAs).
#include "finite.cuh"
#include "umma_util.cuh"

#include <algorithm>
#include <atomic>


namespace sapa {

namespace tma {

using namespace tmau;

constexpr int ROWS = 4, COLS = 8;          // low-res tile of a CTA
constexpr int HH = ROWS + 4;               // halo rows
constexpr int HC = 16;                     // halo columns x0-4 .. x0+11 = one 64-byte row
constexpr int F_KCH = 16;                  // key / query channels per stage (multiple of 8)
constexpr int F_VCH = 32;                  // value channels per stage (multiple of 16)
constexpr int NSTAGE = 4;                  // ring slots of 16 KB
constexpr int NT = 2 * ROWS * 32;          // 8 warps: (row, 4-pixel half)
constexpr int ROWB = HC * 4;               // 64 bytes
constexpr int K_BYTES = HH * F_KCH * ROWB;   // 8192: key box [8 rows][16 ch][16 cols]
constexpr int V_BYTES = HH * F_VCH * ROWB;   // 16384
constexpr int SLOT_BYTES = V_BYTES > 2 * K_BYTES ? V_BYTES : 2 * K_BYTES;   // a key stage = key box + query box of K_BYTES each
constexpr int O_BYTES = 2 * ROWS * F_VCH * ROWB;   // 16384: output box [8 hi rows][32 ch][16 hi cols], double-buffered
constexpr int CTAS_PER_SM = 2;             // resident CTAs per SM the register budget is tuned for

__device__ int g_wait_timeout = 0;         // set when a bounded wait gave up (read by tma_wait_timeout_flag)
// Dynamic tile scheduler of the persistent grid.  Every launch uses one of SCHED_SLOTS counter pairs (chosen
// round-robin on the host); the last CTA of a launch to exit resets its pair, so a pair is clean again long
// before the round-robin comes back to it (that would need SCHED_SLOTS launches resident at the same time).
__device__ unsigned g_next_tile[SCHED_SLOTS];
__device__ unsigned g_ctas_done[SCHED_SLOTS];

// kernel modes: the fused forward, stage 1 of the fused backward, and the two separate ops of the reference's API
constexpr int MODE_FWD = 0;    // out = atn(softmax(sim(query, key)), value); attn = optional softmax output
constexpr int MODE_BWD = 1;    // see the float32 kernel
constexpr int MODE_SIM = 2;    // logits only: attn (output) = sim(query, key); no value stages
constexpr int MODE_AGG = 3;    // aggregation only: out = atn(attn (input weights), value); no key stages

struct Args {
    const void *q, *k, *v; // the inputs themselves: read by the ragged kernels, which have no tensor maps
    void *out, *attn;      // attn: forward = optional output (softmax), backward = input (saved softmax)
    void *ws;              // backward only: logit gradients [B, 25, 2H, 2W], written for the key-gradient gather
    int B, d, C, H, W;
    int rows, ytop0;
    int y_begin, y_end;    // low-res output rows produced by this launch (a band of [0, H); the whole image except in row-slab calls)
    int tiles_x, tiles_y;  // tiles_y covers the band only
    int csplit, vstages;   // work items per tile, each with `vstages` value stages (its own share of the channels): a problem
                           // with few tiles is spread over more CTAs, which all compute the tile's weights
    int sched_slot;        // index into g_next_tile / g_ctas_done
};

// byte offset of element `col` of a 64-byte row under the 64-byte swizzle: the 16-byte chunk index is XORed with
// bits 7..8 of the row's byte offset, which for channel-minor rows of 64 bytes is (channel >> 1) & 3
__device__ __forceinline__ int swz(int col, int channel) { return ((((col >> 2) ^ (channel >> 1)) & 3) << 4) | ((col & 3) << 2); }

// BWD = false: out = atn(softmax(sim(query, key)), value).
// BWD = true : the first half of the backward pass with the same data flow.  The "query" map is grad_out and the
//              "key" map the value tensor (logits = dA = sim(grad_out, value) over C channels); the middle step is the
//              softmax backward dS = A * (dA - sum_k A_k dA_k) with the saved attention map, stored to `ws`; the
//              "value" map is the key tensor and the output is grad_query = agg(dS, key).
// MODE_SIM / MODE_AGG: the logit half / the aggregation half alone (sapa_qk_forward, sapa_av_forward and the halves of
//              the separate backward ops); the weights of MODE_AGG are read where MODE_BWD reads the attention map.
template <int MODE>
__global__ void __launch_bounds__(NT, CTAS_PER_SM)
sapa_tma_fused_f32_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                          const __grid_constant__ CUtensorMap vmap, const __grid_constant__ CUtensorMap omap, const Args a) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long full_bar[NSTAGE];
    // the swizzle pattern is a function of the absolute shared-memory address: align the ring to 1024 bytes
    const unsigned ring_addr = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned bar_addr = (unsigned)__cvta_generic_to_shared(full_bar);
    const unsigned obuf_addr = ring_addr + NSTAGE * SLOT_BYTES;      // two output staging buffers behind the ring

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wrow = warp >> 1, h = warp & 1;
    const int g = lane >> 2, t = lane & 3;
    const int sW = 2 * a.W;
    const size_t hi_plane = (size_t)(2 * a.H) * sW;
    const int nk = (a.d + F_KCH - 1) / F_KCH, nv = a.vstages, total = nk + nv;
    // Persistent CTA: its first tile is blockIdx.x, further tiles come from a global counter.  The stages of
    // successive tiles form one continuous stream through the ring, so the first stages of the next tile are in
    // flight while the current tile finishes.  tile_ids[ti & 3] = tile of the ti-th tile of this CTA, -1 = none.
    const int ntiles = a.B * a.tiles_x * a.tiles_y * a.csplit;     // work items
    __shared__ int tile_ids[4];

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < NSTAGE; ++i) mbar_init(bar_addr + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    begin_after_previous();

    // Stages are issued in stream order (stage gs goes to slot gs % NSTAGE) by thread 0 only.  The producer keeps its
    // position incrementally: per stage it costs a handful of instructions, which matters because the other seven
    // warps wait for warp 0 at the next barrier.
    bool exhausted = false;
    int p_it = 0, p_ti = 0, p_slot = 0, p_n = 0, p_x0 = 0, p_y0 = 0, p_vb = 0;
    auto issue = [&](int) {
        if (exhausted) return;
        if (p_it == 0) {     // first stage of a tile: claim the tile
            int claimed = (int)blockIdx.x;
            if (p_ti > 0) claimed = (int)(atomicAdd(&g_next_tile[a.sched_slot], 1u) + gridDim.x);
            if (claimed >= ntiles) claimed = -1;
            tile_ids[p_ti & 3] = claimed;
            if (claimed < 0) { exhausted = true; return; }
            p_vb = claimed % a.csplit * nv; claimed /= a.csplit;
            p_x0 = (claimed % a.tiles_x) * COLS; claimed /= a.tiles_x;
            p_y0 = a.y_begin + (claimed % a.tiles_y) * ROWS; claimed /= a.tiles_y;
            p_n = claimed;
        }
        const unsigned slot = ring_addr + p_slot * SLOT_BYTES, bar = bar_addr + 8 * p_slot;
        if (p_it < nk) {
            mbar_expect_tx(bar, 2 * K_BYTES);
            tma_load_4d(slot, &kmap, bar, p_x0 - 4, p_it * F_KCH, a.ytop0 + p_y0 - 2, p_n);
            tma_load_4d(slot + K_BYTES, &qmap, bar, 2 * p_x0, p_it * F_KCH, 2 * p_y0, p_n);
        } else {
            mbar_expect_tx(bar, V_BYTES);
            tma_load_4d(slot, &vmap, bar, p_x0 - 4, (p_vb + p_it - nk) * F_VCH, a.ytop0 + p_y0 - 2, p_n);
        }
        if (++p_it == total) { p_it = 0; ++p_ti; }
        p_slot = (p_slot + 1) % NSTAGE;
    };
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < NSTAGE - 1; ++i) issue(i);
    }

    // Lane (g,t): high-res pixel 8h+g of the tile's 16 columns (both rows); after the logit MMAs it holds the
    // window cells j = 2t, 2t+1 of its half's 8-cell span (halo columns 2 + 4h + j); parent l = g/2, window [l, l+4]
    const int l = g >> 1;
    const bool ok0 = (2 * t >= l) && (2 * t <= l + 4), ok1 = (2 * t + 1 >= l) && (2 * t + 1 <= l + 4);

    // swizzled byte offsets inside a 64-byte row
    //   query A fragment: channels ct, ct+2, pixel 8h+g          key B fragment: channels ct, ct+2, cell g -> column 2+4h+g
    //   value A fragment: channel g (and g+8), cells t and t+4 -> columns 2+4h+t, 6+4h+t
    // k index t of a logit fragment reads channel ct = {0, 1, 4, 5}[t] of the 8-channel step and k index t + 4 reads ct + 2
    // (the same permutation for query and key, so the sum over the 8 channels is unchanged): under the 64-byte swizzle
    // channels 0, 1, 4, 5 start in four different 16-byte bank groups, which makes these loads conflict-free (with the
    // identity order, channels t and t + 2 hit the same banks)
    const int ct = (t & 1) + 4 * (t >> 1);
    const int q_off0 = ct * ROWB + swz(8 * h + g, ct), q_off1 = (ct + 2) * ROWB + swz(8 * h + g, ct + 2);
    const int k_off0 = ct * ROWB + swz(2 + 4 * h + g, ct), k_off1 = (ct + 2) * ROWB + swz(2 + 4 * h + g, ct + 2);
    const int v_offa = g * ROWB + swz(2 + 4 * h + t, g), v_offb = g * ROWB + swz(6 + 4 * h + t, g);
    //   output D fragment: channel g (and g+8), pixels 8h+2t, 8h+2t+1 of high-res rows 2*wrow, 2*wrow+1
    const int o_off = (2 * wrow) * (F_VCH * ROWB) + g * ROWB + swz(8 * h + 2 * t, g);

    float s[5][4];                         // logits, then probabilities: [dy][2 * row + (cell 2t | 2t+1)], the MMA's D fragment
    unsigned phi[2][5][2];                 // B fragments of the aggregation: probabilities of cells (t, t+4); their
                                           // low tf32 terms are derived where they are used (2 ALU ops, 20 registers saved)

    // cells (2t, 2t+1) of the logit fragment -> cells (t, t+4), the k order of the value fragments
    auto realign = [&]() {
        const int src_a = (lane & ~3) | (t >> 1), src_b = src_a + 2;
        const bool odd = t & 1;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {
                const float a0 = __shfl_sync(0xffffffffu, s[dy][2 * r], src_a), a1 = __shfl_sync(0xffffffffu, s[dy][2 * r + 1], src_a);
                const float b0 = __shfl_sync(0xffffffffu, s[dy][2 * r], src_b), b1 = __shfl_sync(0xffffffffu, s[dy][2 * r + 1], src_b);
                phi[r][dy][0] = __float_as_uint(odd ? a1 : a0);
                phi[r][dy][1] = __float_as_uint(odd ? b1 : b0);
            }
    };

    int gs = 0;
    for (int ti = 0;; ++ti) {
    // written by thread 0 at least one barrier earlier (tile 0 is known to everybody)
    int tile = ti == 0 ? (int)blockIdx.x : tile_ids[ti & 3];
    if (tile < 0) break;
    const int vb = tile % a.csplit * nv; tile /= a.csplit;
    const int bx = tile % a.tiles_x; tile /= a.tiles_x;
    const int by = tile % a.tiles_y; tile /= a.tiles_y;
    const int n = tile;
    const int x0 = bx * COLS, y0 = a.y_begin + by * ROWS;
    const int y = y0 + wrow;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int dy = 0; dy < 5; ++dy) s[dy][2 * r] = s[dy][2 * r + 1] = 0.f;

    if (MODE == MODE_AGG) {      // the weights come from memory instead of from the logit stages
        const bool pix_ok = y < a.y_end && x0 + 4 * h + l < a.W;
        const float *ap = static_cast<const float *>(a.attn) + (size_t)n * 25 * hi_plane + (size_t)(2 * y) * sW + 2 * (x0 + 4 * h) + g;
#pragma unroll
        for (int dy = 0; dy < 5; ++dy)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                s[dy][2 * r] = (pix_ok && ok0) ? ap[(size_t)(dy * 5 + 2 * t - l) * hi_plane + (size_t)r * sW] : 0.f;
                s[dy][2 * r + 1] = (pix_ok && ok1) ? ap[(size_t)(dy * 5 + 2 * t + 1 - l) * hi_plane + (size_t)r * sW] : 0.f;
            }
        realign();
    }

    for (int it = 0; it < total; ++it, ++gs) {
        // everyone is done with the slot that is refilled next and has written its output fragment
        __syncthreads();
        if (tid == 0) {
            if (it > nk) {   // the previous stage was a value stage: its output tile is complete in shared memory
                tma_store_4d(&omap, obuf_addr + ((it - nk - 1) & 1) * O_BYTES, 2 * x0, (vb + it - nk - 1) * F_VCH, 2 * y0, n);
                asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
            }
            issue(gs + NSTAGE - 1);
        }
        if (!mbar_wait_bounded(bar_addr + 8 * (gs % NSTAGE), (gs / NSTAGE) & 1)) {
            atomicExch(&g_wait_timeout, 1);
            return;
        }
        const unsigned stage = fresh(ring_addr + (gs % NSTAGE) * SLOT_BYTES);

        if (it < nk) {
            // ------------------------------------------------------------- logits: S[16 px][8 cells] += Qt[16 px][8 ch] K[8 ch][8 cells]
            const unsigned kb = stage + wrow * (F_KCH * ROWB);
            const unsigned qb = stage + K_BYTES + (2 * wrow) * (F_KCH * ROWB);
#pragma unroll
            for (int ks = 0; ks < F_KCH / 8; ++ks) {
                unsigned ah[4], al[4];
                ah[0] = lds32(qb + ks * 8 * ROWB + q_off0);                  // Q[ch t][row 0][px g]
                ah[1] = lds32(qb + F_KCH * ROWB + ks * 8 * ROWB + q_off0);     // Q[ch t][row 1][px g]
                ah[2] = lds32(qb + ks * 8 * ROWB + q_off1);                  // Q[ch t+4][row 0]
                ah[3] = lds32(qb + F_KCH * ROWB + ks * 8 * ROWB + q_off1);     // Q[ch t+4][row 1]
#pragma unroll
                for (int i = 0; i < 4; ++i) al[i] = tf32_lo(ah[i]);
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) {
                    const unsigned b0 = lds32(kb + dy * (F_KCH * ROWB) + ks * 8 * ROWB + k_off0);
                    const unsigned b1 = lds32(kb + dy * (F_KCH * ROWB) + ks * 8 * ROWB + k_off1);
                    mma_tf32(s[dy], ah, b0, b1);
                    mma_tf32(s[dy], al, b0, b1);
                    mma_tf32(s[dy], ah, tf32_lo(b0), tf32_lo(b1));
                }
            }
            if (it == nk - 1 && MODE == MODE_BWD) {
                // softmax backward over the 25 window slots of each pixel (spread over the 4 lanes of a quad)
                const bool pix_ok = y < a.y_end && x0 + 4 * h + l < a.W;
                const size_t poff = (size_t)n * 25 * hi_plane + (size_t)(2 * y) * sW + 2 * (x0 + 4 * h) + g;
                const float *ap = static_cast<const float *>(a.attn) + poff;
                float *wp = static_cast<float *>(a.ws) + poff;
                float av[5][4];
#pragma unroll
                for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        av[dy][2 * r] = (pix_ok && ok0) ? ap[(size_t)(dy * 5 + 2 * t - l) * hi_plane + (size_t)r * sW] : 0.f;
                        av[dy][2 * r + 1] = (pix_ok && ok1) ? ap[(size_t)(dy * 5 + 2 * t + 1 - l) * hi_plane + (size_t)r * sW] : 0.f;
                    }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float dot = 0.f;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) dot += av[dy][2 * r] * s[dy][2 * r] + av[dy][2 * r + 1] * s[dy][2 * r + 1];
                    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
                    dot += __shfl_xor_sync(0xffffffffu, dot, 2);
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        s[dy][2 * r] = av[dy][2 * r] * (s[dy][2 * r] - dot);
                        s[dy][2 * r + 1] = av[dy][2 * r + 1] * (s[dy][2 * r + 1] - dot);
                    }
                }
                if (pix_ok) {
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            if (ok0) wp[(size_t)(dy * 5 + 2 * t - l) * hi_plane + (size_t)r * sW] = s[dy][2 * r];
                            if (ok1) wp[(size_t)(dy * 5 + 2 * t + 1 - l) * hi_plane + (size_t)r * sW] = s[dy][2 * r + 1];
                        }
                }
            }
            if (it == nk - 1 && MODE == MODE_FWD) {
                // softmax over the 25 window slots of each pixel (spread over the 4 lanes of a quad)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float m = -INFINITY;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        if (ok0) m = fmaxf(m, s[dy][2 * r]);
                        if (ok1) m = fmaxf(m, s[dy][2 * r + 1]);
                    }
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                    float z = 0.f;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        s[dy][2 * r] = ok0 ? expf(s[dy][2 * r] - m) : 0.f;
                        s[dy][2 * r + 1] = ok1 ? expf(s[dy][2 * r + 1] - m) : 0.f;
                        z += s[dy][2 * r] + s[dy][2 * r + 1];
                    }
                    z += __shfl_xor_sync(0xffffffffu, z, 1);
                    z += __shfl_xor_sync(0xffffffffu, z, 2);
                    const float inv = 1.f / z;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) { s[dy][2 * r] *= inv; s[dy][2 * r + 1] *= inv; }
                }
            }
            if (it == nk - 1 && (MODE == MODE_FWD || MODE == MODE_SIM)) {      // probabilities, or the raw logits of MODE_SIM
                if (a.attn != nullptr && vb == 0 && y < a.y_end && x0 + 4 * h + l < a.W) {
                    float *an = static_cast<float *>(a.attn) + (size_t)n * 25 * hi_plane + (size_t)(2 * y) * sW + 2 * (x0 + 4 * h) + g;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            if (ok0) an[(size_t)(dy * 5 + 2 * t - l) * hi_plane + (size_t)r * sW] = s[dy][2 * r];
                            if (ok1) an[(size_t)(dy * 5 + 2 * t + 1 - l) * hi_plane + (size_t)r * sW] = s[dy][2 * r + 1];
                        }
                }
            }
            if (it == nk - 1 && MODE != MODE_SIM) realign();
        } else {
            // ------------------------------------------------------------- aggregation: Out[16 ch][8 px] += V[16 ch][8 cells] P[8 cells][8 px]
            const unsigned vbox = stage + wrow * (F_VCH * ROWB);
            float acc[F_VCH / 16][2][4];
#pragma unroll
            for (int b = 0; b < F_VCH / 16; ++b)
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[b][r][i] = 0.f;
            unsigned an[F_VCH / 16][4];                     // fragments of the next window row, loaded one row ahead
            auto load_row = [&](int dy) {
#pragma unroll
                for (int b = 0; b < F_VCH / 16; ++b) {
                    const unsigned p = vbox + dy * (F_VCH * ROWB) + b * 16 * ROWB;
                    an[b][0] = lds32(p + v_offa);                 // V[ch g][cell t]
                    an[b][1] = lds32(p + 8 * ROWB + v_offa);      // V[ch g+8][cell t]
                    an[b][2] = lds32(p + v_offb);                 // V[ch g][cell t+4]
                    an[b][3] = lds32(p + 8 * ROWB + v_offb);      // V[ch g+8][cell t+4]
                }
            };
            load_row(0);
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {
                unsigned ah[F_VCH / 16][4], al[F_VCH / 16][4];
#pragma unroll
                for (int b = 0; b < F_VCH / 16; ++b)
#pragma unroll
                    for (int i = 0; i < 4; ++i) ah[b][i] = an[b][i];
                if (dy < 4) load_row(dy + 1);
#pragma unroll
                for (int b = 0; b < F_VCH / 16; ++b)
#pragma unroll
                    for (int i = 0; i < 4; ++i) al[b][i] = tf32_lo(ah[b][i]);
#pragma unroll
                for (int b = 0; b < F_VCH / 16; ++b)
#pragma unroll
                    for (int r = 0; r < 2; ++r) mma_tf32(acc[b][r], ah[b], phi[r][dy][0], phi[r][dy][1]);
#pragma unroll
                for (int b = 0; b < F_VCH / 16; ++b)
#pragma unroll
                    for (int r = 0; r < 2; ++r) mma_tf32(acc[b][r], al[b], phi[r][dy][0], phi[r][dy][1]);
#pragma unroll
                for (int b = 0; b < F_VCH / 16; ++b)
#pragma unroll
                    for (int r = 0; r < 2; ++r) mma_tf32(acc[b][r], ah[b], tf32_lo(phi[r][dy][0]), tf32_lo(phi[r][dy][1]));
            }
            // D fragment: d0,d1 = Out[ch g][px 2t, 2t+1], d2,d3 = Out[ch g+8][px 2t, 2t+1] -> staging buffer laid out
            // as the output box [hi row][channel][16 hi cols] (64-byte swizzle), stored by TMA after the next barrier
            {
                const unsigned ob = obuf_addr + ((it - nk) & 1) * O_BYTES + o_off;
#pragma unroll
                for (int b = 0; b < F_VCH / 16; ++b)
#pragma unroll
                    for (int half = 0; half < 2; ++half)
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            sts64(ob + r * (F_VCH * ROWB) + (16 * b + 8 * half) * ROWB, acc[b][r][2 * half], acc[b][r][2 * half + 1]);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // make the writes visible to the TMA engine
                // the buffer written two value stages from now is this one: its store must have finished reading it
                if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
            }
        }
    }
    // the tile's last output block
    __syncthreads();
    if (tid == 0 && MODE != MODE_SIM) {
        tma_store_4d(&omap, obuf_addr + ((nv - 1) & 1) * O_BYTES, 2 * x0, (vb + nv - 1) * F_VCH, 2 * y0, n);
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
    }
    }
    if (tid == 0) {
        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");   // all output tiles are written
        if (atomicAdd(&g_ctas_done[a.sched_slot], 1u) == gridDim.x - 1) {   // last CTA out: reset the scheduler slot
            g_next_tile[a.sched_slot] = 0u;
            g_ctas_done[a.sched_slot] = 0u;
        }
    }
}

// ---------------------------------------------------------------------------------- float16 / bfloat16
// Same tile (4 x 8 low-res pixels) and scheduler as the float32 kernel; what differs:
//   * key / value boxes are 24 columns wide and start at x0 - 8, the nearest 16-byte boundary below the halo
//     (window cell j of the tile sits in box column j + 6); rows are 48 bytes, unswizzled: eight consecutive
//     channels start in eight different 16-byte bank groups, so every ldmatrix is conflict-free;
//   * query boxes are [8 high-res rows][channels][16 pixels] with 32-byte rows and the 32-byte swizzle;
//   * a warp owns ONE high-res row (16 pixels = two groups of 8): warp = (low-res row, upper / lower high-res row);
//   * logits are computed TRANSPOSED, S^T[16 box columns][8 pixels] = K^T[16 columns][16 ch] Q[16 ch][8 pixels]
//     (m16n8k16; columns 0-15 for the left pixel group, 8-23 for the right one), so that the same 16 columns are
//     the k dimension of the aggregation Out[16 ch][8 px] += V[16 ch][16 columns] P^T[16 columns][8 px]; the
//     accumulator fragment of S^T becomes the B fragment of that product with one movmatrix (8x8 transpose) per
//     packed register;
//   * all fragments come from ldmatrix: K^T and Q with .trans, V without;
//   * no CTA-wide barrier in the steady state: ring slots are handed back on "empty" mbarriers (one arrival per
//     warp) and refilled by one lane of a ninth, producer-only warp; outputs go from registers to global memory.
namespace h16 {
constexpr int COLS = 8;                         // low-res columns of a CTA tile
constexpr int NSTAGE = 4;                       // ring slots of 20 KB
constexpr int NW = 2 * ROWS;                    // 8 consumer warps
constexpr int NT = (NW + 1) * 32;               // + one producer warp
constexpr int PT = 4 * 32;                      // threads of the four producer warps of the ragged form
constexpr int NT_RAGGED = NW * 32 + PT;
constexpr int CTAS_PER_SM = 2;                  // resident CTAs per SM the register budget is tuned for
constexpr int KCH = 32;                         // key / query channels per stage (k steps of 16 for m16n8k16)
constexpr int VCH = 32;                         // value channels per stage (multiple of 16)
constexpr int BC = 24;                          // key / value box columns
constexpr int KROW = BC * 2;                    // 48 bytes
constexpr int QROW = 32;                        // 16 high-res pixels
constexpr int K_BYTES = HH * KCH * KROW;        // 6144
constexpr int Q_BYTES = 2 * ROWS * KCH * QROW;  // 4096
constexpr int V_BYTES = HH * VCH * KROW;        // 12288
constexpr int SLOT_BYTES = V_BYTES > K_BYTES + Q_BYTES ? V_BYTES : K_BYTES + Q_BYTES;
constexpr int SMEM_BYTES = NSTAGE * SLOT_BYTES + 1024;
static_assert(K_BYTES % 256 == 0 && SLOT_BYTES % 256 == 0, "the swizzled query box needs 256-byte alignment");
}  // namespace h16

// Producer warps of the ragged 16-bit kernel: fill one ring slot with the boxes that TMA would put there (the columns of a
// key / value box that a window can reach: box columns 6 .. 17; the others stay zero from the start of the kernel).  Eight
// threads (six of them working) per box row, one pixel pair each.
// Even W: low-res rows start on 4 bytes: asynchronous 4-byte copies.  Odd W: they start on any 2 bytes: two loads into
// registers one stage ahead (OddBox::load), one shared store per pair (OddBox::store).  High-res rows have an even length
// always.
constexpr int LO_ITEMS = HH * 32 * 8 / h16::PT;
template <typename T>
__device__ __forceinline__ void ragged_lo_box_16(unsigned dst, const T *base /* plane 0 of the image */, int c0, int C, int rows, int W, int y0, int x0, int ptid) {
    const int pair = ptid & 7, x = x0 - 2 + 2 * pair;
    const bool x_ok = pair < 6 && x >= 0 && x < W;
    const size_t plane = (size_t)rows * W;
    if (pair >= 6) return;
#pragma unroll
    for (int i = 0; i < LO_ITEMS; ++i) {
        const int rc = i * (h16::PT / 8) + (ptid >> 3), ch = rc & 31, row = rc >> 5, y = y0 - 2 + row;
        const bool ok = x_ok && c0 + ch < C && y >= 0 && y < rows;
        cp_async4(dst + row * (32 * h16::KROW) + ch * h16::KROW + 12 + 4 * pair, ok ? base + (size_t)(c0 + ch) * plane + (size_t)y * W + x : base, ok);
    }
}
struct OddBox {
    unsigned short lo[LO_ITEMS], hi[LO_ITEMS];
    template <typename T>
    __device__ __forceinline__ void load(const T *base, int c0, int C, int rows, int W, int y0, int x0, int ptid) {
        const int pair = ptid & 7, x = x0 - 2 + 2 * pair;
        const bool lo_ok = pair < 6 && x >= 0 && x < W, hi_ok = pair < 6 && x + 1 >= 0 && x + 1 < W;
        const size_t plane = (size_t)rows * W;
        const unsigned short *b16 = reinterpret_cast<const unsigned short *>(base);
#pragma unroll
        for (int i = 0; i < LO_ITEMS; ++i) {
            const int rc = i * (h16::PT / 8) + (ptid >> 3), ch = rc & 31, row = rc >> 5, y = y0 - 2 + row;
            const bool ok = c0 + ch < C && y >= 0 && y < rows;
            const unsigned short *p = b16 + (size_t)(c0 + ch) * plane + (size_t)y * W + x;
            lo[i] = ok && lo_ok ? *p : (unsigned short)0;
            hi[i] = ok && hi_ok ? p[1] : (unsigned short)0;
        }
    }
    __device__ __forceinline__ void store(unsigned dst, int ptid) const {
        const int pair = ptid & 7;
        if (pair >= 6) return;
#pragma unroll
        for (int i = 0; i < LO_ITEMS; ++i) {
            const int rc = i * (h16::PT / 8) + (ptid >> 3), ch = rc & 31, row = rc >> 5;
            sts32(dst + row * (32 * h16::KROW) + ch * h16::KROW + 12 + 4 * pair, (unsigned)lo[i] | ((unsigned)hi[i] << 16));
        }
    }
};
template <typename T>
__device__ __forceinline__ void ragged_hi_box_16(unsigned dst, const T *base, int c0, int C, int H, int W, int y0, int x0, int ptid) {
    const int sW = 2 * W;
    const size_t plane = (size_t)(2 * H) * sW;
    if (!(W & 1)) {               // high-res rows start on 8 bytes: four pixels per copy
        const int quad = ptid & 3;
#pragma unroll
        for (int i = 0; i < 2 * ROWS * 32 * 4 / h16::PT; ++i) {
            const int rc = i * (h16::PT / 4) + (ptid >> 2), ch = rc & 31, row = rc >> 5;
            const bool ok = x0 + 2 * quad < W && c0 + ch < C && 2 * y0 + row < 2 * H;
            cp_async8(dst + row * (32 * h16::QROW) + ch * h16::QROW + ((((quad >> 1) ^ (ch >> 2)) & 1) << 4) + 8 * (quad & 1),
                      ok ? base + (size_t)(c0 + ch) * plane + (size_t)(2 * y0 + row) * sW + 2 * x0 + 4 * quad : base, ok);
        }
        return;
    }
    const int pair = ptid & 7;
    const bool x_ok = x0 + pair < W;
#pragma unroll
    for (int i = 0; i < 2 * ROWS * 32 * 8 / h16::PT; ++i) {
        const int rc = i * (h16::PT / 8) + (ptid >> 3), ch = rc & 31, row = rc >> 5;
        const bool ok = x_ok && c0 + ch < C && 2 * y0 + row < 2 * H;
        cp_async4(dst + row * (32 * h16::QROW) + ch * h16::QROW + ((((pair >> 2) ^ (ch >> 2)) & 1) << 4) + 4 * (pair & 3),
                  ok ? base + (size_t)(c0 + ch) * plane + (size_t)(2 * y0 + row) * sW + 2 * (x0 + pair) : base, ok);
    }
}

// The sums of a value stage over the 25 cells of every pixel alone, for a warp with a sum that is not finite.  The matrix product
// also takes the other cells of its 16 columns, with weights of zero, and 0 * inf would reach pixels whose window has no
// infinity; of a weight in two terms the second may be negative, and inf - inf would take the place of an infinity inside it.
// WEIGHTS_POSITIVE: softmax weights, of which none is zero however small its 16-bit terms are.
template <typename T, bool TWO, bool WEIGHTS_POSITIVE, int N>
__device__ __forceinline__ void window_sums(float (&acc)[h16::VCH / 16][2][4], const unsigned (&pb)[2][5][2], const unsigned (&pl)[N][5][2], unsigned rows,
                                            int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        float sum[h16::VCH / 16][4] = {};
#pragma unroll
        for (int dy = 0; dy < 5; ++dy)
#pragma unroll 1
            for (int dx = 0; dx < 5; ++dx) {
                // cell k of the 16 lies in the fragment of lane (pixel, (k & 7) / 2), register k / 8, half k & 1
                const int k = 6 + t - 4 * p + dx;
                float w[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int src = 4 * (2 * t + j) + ((k & 7) >> 1);
                    const auto term = [&](unsigned left, unsigned right) {
                        const unsigned l = __shfl_sync(0xffffffffu, left, src), r = __shfl_sync(0xffffffffu, right, src);
                        const float2 f = unpack_pair(T(), k & 8 ? r : l);
                        return k & 1 ? f.y : f.x;
                    };
                    w[j] = term(pb[p][dy][0], pb[p][dy][1]);
                    if constexpr (TWO) {
                        const float second = term(pl[p][dy][0], pl[p][dy][1]);
                        if (fabsf(w[j]) <= FLT_MAX) w[j] += second;
                    }
                    if (WEIGHTS_POSITIVE && w[j] == 0.f) w[j] = FLT_MIN;
                }
                const unsigned cell = rows + (dy * h16::VCH + g) * h16::KROW + 2 * (8 * p + k);
#pragma unroll
                for (int i = 0; i < h16::VCH / 8; ++i) {       // channel g + 8i: block i/2, half i%2
                    const float v = lds_16(T(), cell + 8 * i * h16::KROW);
                    sum[i >> 1][2 * (i & 1)] = fmaf(w[0], v, sum[i >> 1][2 * (i & 1)]);
                    sum[i >> 1][2 * (i & 1) + 1] = fmaf(w[1], v, sum[i >> 1][2 * (i & 1) + 1]);
                }
            }
#pragma unroll
        for (int b = 0; b < h16::VCH / 16; ++b)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[b][p][i] = sum[b][i];
    }
}

// modes: see the float32 kernel.  RAGGED: rows that are not multiples of 16 bytes - no tensor maps, four producer warps copy
// the boxes (static tile order); everything behind the ring is the same.  The FP32-pipe kernels it replaced walked all
// channels in one CTA per 4 x 32 tile: backward of B=2, C=256, d=32, 25x42 -> 50x84 in bfloat16 438 -> 60 us.  At large
// sizes the copies bound it: 1.7 - 2x the time of the neighbouring aligned width (8 x 256 x 64x65: 110 us, 64x64: 56 us).
template <typename T, int MODE, bool RAGGED>
__global__ void __launch_bounds__(RAGGED ? h16::NT_RAGGED : h16::NT, RAGGED ? 1 : h16::CTAS_PER_SM)
sapa_tma_fused_16_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                         const __grid_constant__ CUtensorMap vmap, const Args a) {
    using namespace h16;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * h16::NSTAGE];      // full[NSTAGE], empty[NSTAGE]
    __shared__ int tile_ids[4];       // tile_ids[ti & 3] = tile of the ti-th tile of this CTA, -1 = no more tiles
    const unsigned ring_addr = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned full_addr = (unsigned)__cvta_generic_to_shared(bars), empty_addr = full_addr + 8 * h16::NSTAGE;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wrow = warp >> 1, r = warp & 1;
    const int g = lane >> 2, t = lane & 3;
    const int sW = 2 * a.W;
    const size_t hi_plane = (size_t)(2 * a.H) * sW;
    const int nk = (a.d + KCH - 1) / KCH, nv = a.vstages, total = nk + nv;
    const int ntiles = a.B * a.tiles_x * a.tiles_y * a.csplit;     // work items

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < h16::NSTAGE; ++i) {
            mbar_init(full_addr + 8 * i, RAGGED ? (a.W & 1 ? 2 * PT : PT) : 1);
            mbar_init(empty_addr + 8 * i, NW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if constexpr (RAGGED)       // box columns that are never copied must read as zero
        for (int i = tid; i < h16::NSTAGE * h16::SLOT_BYTES / 4; i += h16::NT_RAGGED) sts32(ring_addr + 4 * i, 0u);
    __syncthreads();
    begin_after_previous();

    if constexpr (RAGGED) {
        if (warp >= NW) {
            const int ptid = tid - NW * 32;
            const T *qp = static_cast<const T *>(a.q), *kp = static_cast<const T *>(a.k), *vp = static_cast<const T *>(a.v);
            const size_t lo_plane = (size_t)a.rows * a.W;
            // position of a stage: its low-res box is read one stage ahead when W is odd
            struct Pos { int tile, it, x0, y0, n, vb; };
            const auto locate = [&](Pos &p) {
                int t_ = p.tile / a.csplit;
                p.vb = p.tile % a.csplit * nv;
                p.x0 = (t_ % a.tiles_x) * h16::COLS; t_ /= a.tiles_x;
                p.y0 = a.y_begin + (t_ % a.tiles_y) * ROWS; p.n = t_ / a.tiles_y;
            };
            const auto advance = [&](Pos &p) {
                if (++p.it < total) return;
                p.it = 0;
                p.tile += gridDim.x;
                if (p.tile < ntiles) locate(p);
            };
            Pos cur{(int)blockIdx.x, 0, 0, 0, 0, 0};
            locate(cur);
            int slot = 0, phase = 0;
            const auto claim = [&]() {
                if (mbar_wait_bounded(empty_addr + 8 * slot, phase ^ 1)) return true;
                atomicExch(&g_wait_timeout, 1);
                cp_async_wait_all();
                return false;
            };
            const auto next_slot = [&]() { if (++slot == h16::NSTAGE) { slot = 0; phase ^= 1; } };
            if (MODE == MODE_FWD || (a.W & 1)) {      // rows of even length have another forward kernel
                OddBox box;
                const auto load = [&](const Pos &p) {
                    const bool key = p.it < nk;
                    box.load(key ? kp + (size_t)p.n * a.d * lo_plane : vp + (size_t)p.n * a.C * lo_plane, key ? p.it * KCH : (p.vb + p.it - nk) * VCH,
                             key ? a.d : a.C, a.rows, a.W, a.ytop0 + p.y0, p.x0, ptid);
                };
                load(cur);
                while (cur.tile < ntiles) {
                    if (!claim()) return;
                    const unsigned dst = ring_addr + slot * h16::SLOT_BYTES, bar = full_addr + 8 * slot;
                    if (cur.it < nk) ragged_hi_box_16<T>(dst + h16::K_BYTES, qp + (size_t)cur.n * a.d * hi_plane, cur.it * KCH, a.d, a.H, a.W, cur.y0, cur.x0, ptid);
                    box.store(dst, ptid);
                    cp_async_arrive(bar);        // the query copies, and ...
                    mbar_arrive(bar);            // ... the shared stores (two arrivals per thread)
                    next_slot();
                    advance(cur);
                    if (cur.tile < ntiles) load(cur);
                }
            } else {
                while (cur.tile < ntiles) {
                    if (!claim()) return;
                    const unsigned dst = ring_addr + slot * h16::SLOT_BYTES;
                    const bool key = cur.it < nk;
                    ragged_lo_box_16<T>(dst, key ? kp + (size_t)cur.n * a.d * lo_plane : vp + (size_t)cur.n * a.C * lo_plane,
                                        key ? cur.it * KCH : (cur.vb + cur.it - nk) * VCH, key ? a.d : a.C, a.rows, a.W, a.ytop0 + cur.y0, cur.x0, ptid);
                    if (key) ragged_hi_box_16<T>(dst + h16::K_BYTES, qp + (size_t)cur.n * a.d * hi_plane, cur.it * KCH, a.d, a.H, a.W, cur.y0, cur.x0, ptid);
                    cp_async_arrive(full_addr + 8 * slot);
                    next_slot();
                    advance(cur);
                }
            }
            cp_async_wait_all();
            return;
        }
    }

    // ---- producer state (lane 0 of the producer warp).  The stages of successive tiles form one continuous stream through
    // the ring; the first tile of a CTA is blockIdx.x, further tiles come from a global counter.
    int p_issued = 0, p_slot = 0, p_phase = 0, p_it = 0, p_ti = 0, p_n = 0, p_x0 = 0, p_y0 = 0, p_vb = 0;
    bool p_done = false;
    // Issues every stage whose slot is free; when the stage `need` (the one the warp is about to wait for) has not
    // been issued yet it waits for that slot.  A slot is free when all NW warps have released its previous use; on
    // a fresh barrier the wait for the parity of the "previous" phase succeeds at once.
    auto produce = [&](int need) {
        while (!p_done) {
            const unsigned ebar = empty_addr + 8 * p_slot;
            if (!mbar_test_wait(ebar, p_phase ^ 1)) {
                if (p_issued > need) return;
                if (!mbar_wait_bounded(ebar, p_phase ^ 1)) {
                    atomicExch(&g_wait_timeout, 1);
                    p_done = true;
                    return;
                }
            }
            const unsigned bar = full_addr + 8 * p_slot;
            if (p_it == 0) {
                int claimed = (int)blockIdx.x;
                if (p_ti > 0) claimed = (int)(atomicAdd(&g_next_tile[a.sched_slot], 1u) + gridDim.x);
                if (claimed >= ntiles) claimed = -1;
                tile_ids[p_ti & 3] = claimed;
                if (claimed < 0) {
                    mbar_arrive(bar);          // completes the phase without data: the warps read -1 and stop
                    if (atomicAdd(&g_ctas_done[a.sched_slot], 1u) == gridDim.x - 1) {   // last CTA out: reset the scheduler slot
                        g_next_tile[a.sched_slot] = 0u;
                        g_ctas_done[a.sched_slot] = 0u;
                    }
                    p_done = true;
                    return;
                }
                p_vb = claimed % a.csplit * nv; claimed /= a.csplit;
                p_x0 = (claimed % a.tiles_x) * h16::COLS; claimed /= a.tiles_x;
                p_y0 = a.y_begin + (claimed % a.tiles_y) * ROWS; claimed /= a.tiles_y;
                p_n = claimed;
            }
            const unsigned dst = ring_addr + p_slot * h16::SLOT_BYTES;
            if (p_it < nk) {
                mbar_expect_tx(bar, h16::K_BYTES + Q_BYTES);
                tma_load_4d(dst, &kmap, bar, p_x0 - 8, p_it * KCH, a.ytop0 + p_y0 - 2, p_n);
                tma_load_4d(dst + h16::K_BYTES, &qmap, bar, 2 * p_x0, p_it * KCH, 2 * p_y0, p_n);
            } else {
                mbar_expect_tx(bar, h16::V_BYTES);
                tma_load_4d(dst, &vmap, bar, p_x0 - 8, (p_vb + p_it - nk) * VCH, a.ytop0 + p_y0 - 2, p_n);
            }
            ++p_issued;
            if (++p_it == total) { p_it = 0; ++p_ti; }
            if (++p_slot == h16::NSTAGE) { p_slot = 0; p_phase ^= 1; }
        }
    };

    // The producer is a warp of its own (one lane works): inside a consumer warp it sat on that warp's critical path -
    // 40 % of the warp's time at config 2 - and the other warps waited for the stages it had not issued yet.
    if (!RAGGED && warp == NW) {
        if (lane == 0) produce(0x7fffffff);
        return;
    }

    // ---- per-lane constants
    // ldmatrix row addresses.  "A-type" lane order: matrices (rows 0-7 | 8-15) x (chunk 0 | 1) as m0..m3 =
    // (lo,0) (hi,0) (lo,1) (hi,1); "T-type": (lo,0) (lo,1) (hi,0) (hi,1).
    const int row_a = (lane & 7) + 8 * ((lane >> 3) & 1), chunk_a = lane >> 4;
    const int row_t = (lane & 7) + 8 * (lane >> 4), chunk_t = (lane >> 3) & 1;
    // query (B of the logits): m0..m3 = (ch 0-7, px 0-7) (ch 8-15, px 0-7) (ch 0-7, px 8-15) (ch 8-15, px 8-15)
    const int q_off = h16::K_BYTES + (2 * wrow + r) * (KCH * QROW) + row_a * QROW + (((chunk_a ^ (row_a >> 2)) & 1) << 4);
    // key (A of the logits, transposed): m0..m3 = (ch 0-7, col 0-7) (ch 0-7, col 8-15) (ch 8-15, col 0-7) (ch 8-15, col 8-15),
    // then m4, m5 = (ch 0-7, col 16-23) (ch 8-15, col 16-23).  The right pixel group's fragment is assembled from
    // m1, m4, m3, m5 (the shared middle columns are loaded once: the kernel is short of shared-memory bandwidth, not of
    // issue slots).
    const int k_off = wrow * (KCH * KROW) + row_t * KROW + chunk_t * 16;
    const int k_off2 = wrow * (KCH * KROW) + row_a * KROW + 32;
    // value (A of the aggregation): m0..m3 = (ch 0-7, col 0-7) (ch 8-15, col 0-7) (ch 0-7, col 8-15) (ch 8-15, col 8-15),
    // then m4, m5 = (ch 0-7, col 16-23) (ch 8-15, col 16-23)
    const int v_off = wrow * (VCH * KROW) + row_a * KROW + chunk_a * 16;
    const int v_off2 = wrow * (VCH * KROW) + row_a * KROW + 32;
    // Lane (g,t) of pixel group p (pixels 8p .. 8p+7 of the row) holds, for the pixels 8p+2t and 8p+2t+1 (parent
    // column l = 4p + t, window = box columns l+6 .. l+10), the box columns 8p+g ("lo") and 8p+g+8 ("hi").
    bool ok_lo[2], ok_hi[2];
    int dx_lo[2];                 // window column of the lo cell (hi = lo + 8)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        dx_lo[p] = 4 * p + g - t - 6;
        ok_lo[p] = dx_lo[p] >= 0 && dx_lo[p] <= 4;
        ok_hi[p] = dx_lo[p] + 8 >= 0 && dx_lo[p] + 8 <= 4;
    }

    float s[2][5][4];             // logits, then probabilities: [group][dy][(lo,px0) (lo,px1) (hi,px0) (hi,px1)]
    unsigned pb[2][5][2];         // B fragments of the aggregation
    // Rows of any length: the FP32-pipe kernels that served them kept the weights in float32, so here they are two terms (pb + pl, 16
    // bits of a bfloat16 pair, 22 of a float16 one).  Logit gradients have no fixed range: each pixel's are scaled by a power of
    // two to [1, 2) before they are split, its outputs are scaled back.
    constexpr bool TWO = RAGGED && (MODE == MODE_FWD || MODE == MODE_BWD);
    unsigned pl[TWO ? 2 : 1][5][2];
    float back[2][2] = {{1.f, 1.f}, {1.f, 1.f}};
    const auto two_terms = [&](float x, float y, unsigned &hi, unsigned &lo) {
        hi = pack_pair(T(), x, y);
        const float2 f = unpack_pair(T(), hi);
        lo = pack_pair(T(), x - f.x, y - f.y);
    };

    int slot = 0, phase = 0, it = 0, ti = 0, gs = 0;
    int n = 0, x0 = 0, y = 0;
    int c0 = 0;                   // first channel of the current value stage
    // kernel-wide strides in 32-bit words of the 16-bit output / attention tensors (two elements per word)
    const size_t plane_w = hi_plane >> 1;
    const int C = a.C, Wlo = a.W;
    unsigned *o_ptr = nullptr;            // this lane's output word for the first channel of the current value stage
    bool row_ok = false, col_ok0 = false, col_ok1 = false;
    constexpr float LOG2E = 1.4426950408889634f;
    for (;; ++gs) {
        if (RAGGED && it == 0 && (int)blockIdx.x + ti * (int)gridDim.x >= ntiles) break;
        if (!mbar_wait_bounded(full_addr + 8 * slot, phase)) {
            atomicExch(&g_wait_timeout, 1);
            return;
        }
        if (it == 0) {
            int tile = RAGGED ? (int)blockIdx.x + ti * (int)gridDim.x : tile_ids[ti & 3];      // published by the producer before the barrier's phase completed
            if (tile < 0) break;
            c0 = tile % a.csplit * nv * VCH; tile /= a.csplit;
            x0 = (tile % a.tiles_x) * h16::COLS; tile /= a.tiles_x;
            y = a.y_begin + (tile % a.tiles_y) * ROWS + wrow; tile /= a.tiles_y;
            n = tile;
            row_ok = y < a.y_end; col_ok0 = x0 + t < Wlo; col_ok1 = x0 + 4 + t < Wlo;
            o_ptr = reinterpret_cast<unsigned *>(static_cast<T *>(a.out) + ((size_t)n * C + c0 + g) * hi_plane +
                                                 (size_t)(2 * y + r) * sW + 2 * x0 + 2 * t);
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[p][dy][i] = 0.f;
        }
        if (MODE == MODE_AGG && it == 0) {      // the weights come from memory, already in the packed pair layout
            const unsigned *ap = static_cast<const unsigned *>(a.attn) +
                                 (((size_t)n * 25 * hi_plane + (size_t)(2 * y + r) * sW + 2 * x0 + 2 * t) >> 1);
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const bool pix = row_ok && (p == 0 ? col_ok0 : col_ok1);
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) {
                    unsigned ulo = 0u, uhi = 0u;
                    if (pix && ok_lo[p]) ulo = ap[(size_t)(dy * 5 + dx_lo[p]) * plane_w + 4 * p];
                    if (pix && ok_hi[p]) uhi = ap[(size_t)(dy * 5 + dx_lo[p] + 8) * plane_w + 4 * p];
                    pb[p][dy][0] = movmatrix_trans(ulo);
                    pb[p][dy][1] = movmatrix_trans(uhi);
                }
            }
        }
        const unsigned stage = fresh(ring_addr + slot * h16::SLOT_BYTES);

        if (it < nk) {
            // ------------------------------------------------------------- logits
#pragma unroll
            for (int ks = 0; ks < KCH / 16; ++ks) {
                unsigned qb[4];
                ldsm_x4_trans(qb, stage + q_off + ks * 16 * QROW);
                const unsigned ka_addr = stage + k_off + ks * 16 * KROW, kc_addr = stage + k_off2 + ks * 16 * KROW;
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) {
                    unsigned ka[4], kc[2];
                    ldsm_x4_trans(ka, ka_addr + dy * (KCH * KROW));
                    ldsm_x2_trans(kc, kc_addr + dy * (KCH * KROW));
                    mma_h16<T>(s[0][dy], ka[0], ka[1], ka[2], ka[3], qb[0], qb[1]);
                    mma_h16<T>(s[1][dy], ka[1], kc[0], ka[3], kc[1], qb[2], qb[3]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_addr + 8 * slot);
            if (it == nk - 1 && MODE == MODE_BWD) {
                // softmax backward; the saved attention map is read and the logit gradients are written as 32-bit
                // pairs (the two pixels of a lane are neighbours in memory)
                const size_t poff = ((size_t)n * 25 * hi_plane + (size_t)(2 * y + r) * sW + 2 * x0 + 2 * t) >> 1;
                const unsigned *ap = static_cast<const unsigned *>(a.attn) + poff;
                unsigned *wp = static_cast<unsigned *>(a.ws) + poff;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const bool pix = row_ok && (p == 0 ? col_ok0 : col_ok1);
                    if constexpr (RAGGED)          // cells outside the window may hold an infinity: 0 * inf in the sums below
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            if (!ok_lo[p]) s[p][dy][0] = s[p][dy][1] = 0.f;
                            if (!ok_hi[p]) s[p][dy][2] = s[p][dy][3] = 0.f;
                        }
                    float av[5][4];
                    float d0 = 0.f, d1 = 0.f;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        unsigned ulo = 0u, uhi = 0u;
                        if (pix && ok_lo[p]) ulo = ap[(size_t)(dy * 5 + dx_lo[p]) * plane_w + 4 * p];
                        if (pix && ok_hi[p]) uhi = ap[(size_t)(dy * 5 + dx_lo[p] + 8) * plane_w + 4 * p];
                        const float2 flo = unpack_pair(T(), ulo), fhi = unpack_pair(T(), uhi);
                        av[dy][0] = flo.x; av[dy][1] = flo.y; av[dy][2] = fhi.x; av[dy][3] = fhi.y;
                        d0 += av[dy][0] * s[p][dy][0] + av[dy][2] * s[p][dy][2];
                        d1 += av[dy][1] * s[p][dy][1] + av[dy][3] * s[p][dy][3];
                    }
#pragma unroll
                    for (int sh = 4; sh < 32; sh <<= 1) {
                        d0 += __shfl_xor_sync(0xffffffffu, d0, sh);
                        d1 += __shfl_xor_sync(0xffffffffu, d1, sh);
                    }
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        pb[p][dy][0] = pack_pair(T(), av[dy][0] * (s[p][dy][0] - d0), av[dy][1] * (s[p][dy][1] - d1));
                        pb[p][dy][1] = pack_pair(T(), av[dy][2] * (s[p][dy][2] - d0), av[dy][3] * (s[p][dy][3] - d1));
                        if (pix && ok_lo[p]) wp[(size_t)(dy * 5 + dx_lo[p]) * plane_w + 4 * p] = pb[p][dy][0];
                        if (pix && ok_hi[p]) wp[(size_t)(dy * 5 + dx_lo[p] + 8) * plane_w + 4 * p] = pb[p][dy][1];
                    }
                    if constexpr (TWO) {
                        float m0 = 0.f, m1 = 0.f;
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            av[dy][0] *= s[p][dy][0] - d0; av[dy][1] *= s[p][dy][1] - d1;
                            av[dy][2] *= s[p][dy][2] - d0; av[dy][3] *= s[p][dy][3] - d1;
                            m0 = fmaxf(m0, fmaxf(fabsf(av[dy][0]), fabsf(av[dy][2])));
                            m1 = fmaxf(m1, fmaxf(fabsf(av[dy][1]), fabsf(av[dy][3])));
                        }
#pragma unroll
                        for (int sh = 4; sh < 32; sh <<= 1) {
                            m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, sh));
                            m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, sh));
                        }
                        const int e0 = min(max(254 - (int)(__float_as_uint(m0) >> 23), 1), 253), e1 = min(max(254 - (int)(__float_as_uint(m1) >> 23), 1), 253);
                        const float f0 = __uint_as_float(e0 << 23), f1 = __uint_as_float(e1 << 23);
                        back[p][0] = __uint_as_float((254 - e0) << 23); back[p][1] = __uint_as_float((254 - e1) << 23);
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            two_terms(av[dy][0] * f0, av[dy][1] * f1, pb[p][dy][0], pl[p][dy][0]);
                            two_terms(av[dy][2] * f0, av[dy][3] * f1, pb[p][dy][1], pl[p][dy][1]);
                        }
                    }
                }
            }
            if (it == nk - 1 && MODE == MODE_FWD) {
                // softmax over the 25 window slots of each pixel: 5 rows here x the lanes with the same t.
                // exp(x - m) = 2^(x * log2(e) - m * log2(e)): one FMA and one ex2 per element.
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        if (ok_lo[p]) { m0 = fmaxf(m0, s[p][dy][0]); m1 = fmaxf(m1, s[p][dy][1]); }
                        if (ok_hi[p]) { m0 = fmaxf(m0, s[p][dy][2]); m1 = fmaxf(m1, s[p][dy][3]); }
                    }
#pragma unroll
                    for (int sh = 4; sh < 32; sh <<= 1) {
                        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, sh));
                        m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, sh));
                    }
                    m0 *= LOG2E; m1 *= LOG2E;
                    float z0 = 0.f, z1 = 0.f;
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        s[p][dy][0] = ok_lo[p] ? ex2_ftz(fmaf(s[p][dy][0], LOG2E, -m0)) : 0.f;
                        s[p][dy][1] = ok_lo[p] ? ex2_ftz(fmaf(s[p][dy][1], LOG2E, -m1)) : 0.f;
                        s[p][dy][2] = ok_hi[p] ? ex2_ftz(fmaf(s[p][dy][2], LOG2E, -m0)) : 0.f;
                        s[p][dy][3] = ok_hi[p] ? ex2_ftz(fmaf(s[p][dy][3], LOG2E, -m1)) : 0.f;
                        z0 += s[p][dy][0] + s[p][dy][2];
                        z1 += s[p][dy][1] + s[p][dy][3];
                    }
#pragma unroll
                    for (int sh = 4; sh < 32; sh <<= 1) {
                        z0 += __shfl_xor_sync(0xffffffffu, z0, sh);
                        z1 += __shfl_xor_sync(0xffffffffu, z1, sh);
                    }
                    const float i0 = __frcp_rn(z0), i1 = __frcp_rn(z1);
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        if constexpr (TWO) {
                            two_terms(s[p][dy][0] * i0, s[p][dy][1] * i1, pb[p][dy][0], pl[p][dy][0]);
                            two_terms(s[p][dy][2] * i0, s[p][dy][3] * i1, pb[p][dy][1], pl[p][dy][1]);
                        } else {
                            pb[p][dy][0] = pack_pair(T(), s[p][dy][0] * i0, s[p][dy][1] * i1);
                            pb[p][dy][1] = pack_pair(T(), s[p][dy][2] * i0, s[p][dy][3] * i1);
                        }
                    }
                }
            }
            if (it == nk - 1 && MODE == MODE_SIM) {      // raw logits
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        pb[p][dy][0] = pack_pair(T(), s[p][dy][0], s[p][dy][1]);
                        pb[p][dy][1] = pack_pair(T(), s[p][dy][2], s[p][dy][3]);
                    }
            }
            if (it == nk - 1 && (MODE == MODE_FWD || MODE == MODE_SIM)) {
                if (a.attn != nullptr && c0 == 0 && row_ok) {
                    // the two pixels of a pair are neighbours in memory: one 32-bit store per (window slot, pair)
                    unsigned *an = reinterpret_cast<unsigned *>(static_cast<T *>(a.attn) + (size_t)n * 25 * hi_plane +
                                                                (size_t)(2 * y + r) * sW + 2 * x0 + 2 * t);
#pragma unroll
                    for (int p = 0; p < 2; ++p)
                        if (p == 0 ? col_ok0 : col_ok1) {
#pragma unroll
                            for (int dy = 0; dy < 5; ++dy) {
                                if (ok_lo[p]) an[(size_t)(dy * 5 + dx_lo[p]) * plane_w + 4 * p] = pb[p][dy][0];
                                if (ok_hi[p]) an[(size_t)(dy * 5 + dx_lo[p] + 8) * plane_w + 4 * p] = pb[p][dy][1];
                            }
                        }
                }
            }
            if (it == nk - 1 && MODE != MODE_SIM) {
                // S^T accumulator fragments -> B fragments of the aggregation
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        pb[p][dy][0] = movmatrix_trans(pb[p][dy][0]);
                        pb[p][dy][1] = movmatrix_trans(pb[p][dy][1]);
                        if constexpr (TWO) {
                            pl[p][dy][0] = movmatrix_trans(pl[p][dy][0]);
                            pl[p][dy][1] = movmatrix_trans(pl[p][dy][1]);
                        }
                    }
            }
        } else {
            // ------------------------------------------------------------- aggregation
            float acc[VCH / 16][2][4];
#pragma unroll
            for (int b = 0; b < VCH / 16; ++b)
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[b][p][i] = 0.f;
            const unsigned va_addr = stage + v_off, vc_addr = stage + v_off2;
#pragma unroll
            for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                for (int b = 0; b < VCH / 16; ++b) {
                    unsigned va[4], vc[2];
                    ldsm_x4(va, va_addr + dy * (VCH * KROW) + b * 16 * KROW);
                    ldsm_x2(vc, vc_addr + dy * (VCH * KROW) + b * 16 * KROW);
                    mma_h16<T>(acc[b][0], va[0], va[1], va[2], va[3], pb[0][dy][0], pb[0][dy][1]);
                    mma_h16<T>(acc[b][1], va[2], va[3], vc[0], vc[1], pb[1][dy][0], pb[1][dy][1]);
                    if constexpr (TWO) {
                        mma_h16<T>(acc[b][0], va[0], va[1], va[2], va[3], pl[0][dy][0], pl[0][dy][1]);
                        mma_h16<T>(acc[b][1], va[2], va[3], vc[0], vc[1], pl[1][dy][0], pl[1][dy][1]);
                    }
                }
            if constexpr (RAGGED) {
                float zero[4] = {};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int b = 0; b < VCH / 16; ++b)
#pragma unroll
                        for (int p = 0; p < 2; ++p) zero[i] = fmaf(acc[b][p][i], 0.f, zero[i]);
                if (__any_sync(0xffffffffu, !((zero[0] + zero[1]) + (zero[2] + zero[3]) == 0.f)))
                    window_sums<T, TWO, MODE == MODE_FWD>(acc, pb, pl, stage + wrow * (VCH * KROW), lane);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_addr + 8 * slot);
            // D fragment of group p: d0,d1 = Out[ch g][px 8p+2t, +1], d2,d3 = Out[ch g+8][same].  Neighbouring lanes swap one
            // pair so that even lanes hold pixels 2t .. 2t+3 of the left group and odd lanes 2(t-1) .. 2(t-1)+3 of the right
            // group: a quad then writes one full 32-byte sector per store instruction (half sectors cost an L1 tag cycle each).
            unsigned *o = o_ptr + ((t & 1) ? 3 : 0);
            o_ptr += (size_t)VCH * plane_w;
            if (row_ok) {          // warp-uniform; columns are always inside (W is a multiple of the tile width here)
                const bool odd = t & 1;
#pragma unroll
                for (int j = 0; j < VCH / 8; ++j) {       // channel g + 8j: block j/2, half j%2
                    if constexpr (TWO && MODE == MODE_BWD)
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            acc[j >> 1][p][2 * (j & 1)] *= back[p][0];
                            acc[j >> 1][p][2 * (j & 1) + 1] *= back[p][1];
                        }
                    const unsigned v0 = pack_pair(T(), acc[j >> 1][0][2 * (j & 1)], acc[j >> 1][0][2 * (j & 1) + 1]);
                    const unsigned v1 = pack_pair(T(), acc[j >> 1][1][2 * (j & 1)], acc[j >> 1][1][2 * (j & 1) + 1]);
                    if constexpr (RAGGED) {       // rows on 4-byte boundaries, columns to be checked: one pair per store
                        unsigned *oc = o - (odd ? 3 : 0);
                        if (c0 + 8 * j + g < C) {
                            if (col_ok0) oc[0] = v0;
                            if (col_ok1) oc[4] = v1;
                        }
                        o += 8 * plane_w;
                        continue;
                    }
                    const unsigned got = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
                    if (c0 + 8 * j + g < C) __stcs(reinterpret_cast<uint2 *>(o), odd ? make_uint2(got, v1) : make_uint2(v0, got));
                    o += 8 * plane_w;
                }
            }
            c0 += VCH;
        }
        if (++slot == h16::NSTAGE) { slot = 0; phase ^= 1; }
        if (++it == total) { it = 0; ++ti; }
    }
}

#include "sapa_wide16.cuh"
#include "sapa_strip.cuh"
#include "sapa_strip_fwd.cuh"
#include "sapa_strip_sim.cuh"
#include "sapa_strip_sim16.cuh"

// ---------------------------------------------------------------------------------- host side
// one host-side counter for every kernel of this file: they all share g_next_tile / g_ctas_done, so two launches that
// may be in flight together (different streams, different kernels) must never get the same slot
static std::atomic<unsigned> g_next_sched_slot{0}, g_next_captured_slot{0};

// Opts in to the dynamic shared memory, sizes the persistent grid, picks a scheduler slot and launches.
template <typename Kernel, typename... Maps>
static int launch_persistent(Kernel kernel, const char *name, int threads, int smem, int ctas_per_sm, bool split, Args &a, cudaStream_t st,
                             const Maps &...maps) {
    long long nblocks = (long long)a.B * a.tiles_x * a.tiles_y;
    if (nblocks > 0x7fffffffLL) {
        set_error("too many tiles");
        return SAPA_ERR_ARGUMENT;
    }
    int sms = 0;
    if (int e = prepare_launch(reinterpret_cast<const void *>(kernel), smem, name, sms)) return e;
    const long long resident = (long long)ctas_per_sm * sms;
    // halve the channels of an item as long as all items still run at once (stage 1 of the backward writes its logit
    // gradients and has one or two value stages: not split)
    while (split && a.vstages >= 2 && a.vstages % 2 == 0 && 2 * nblocks <= resident) {
        a.vstages /= 2;
        a.csplit *= 2;
        nblocks *= 2;
    }
    // persistent grid with dynamic tile claiming (static striding left SMs with 6 to 8 tiles instead of ~6.9)
    const unsigned grid = (unsigned)(nblocks < resident ? nblocks : resident);
    a.sched_slot = next_sched_slot(g_next_sched_slot, g_next_captured_slot, st);
    launch_next(kernel, grid, threads, smem, st, maps..., a);
    return check_launch(name);
}

// The strip kernel's split of a problem: rows of an item for the fewest steps (low-res rows) of the busiest CTA, one more for an item's
// halo rows and three to start.
struct StripPlan { strip::SArgs a; long long items, steps; };
template <typename T> static StripPlan strip_plan(int B, int C, int H, int W, int rows, int ytop0, int y_begin, int y_end, int sms) {
    StripPlan p{};
    strip::SArgs &a = p.a;
    a.B = B; a.C = C; a.H = H; a.W = W; a.rows = rows; a.ytop0 = ytop0; a.y_begin = y_begin; a.y_end = y_end;
    a.wrows = H; a.wy0 = 0;
    a.strips = ceil_div(W, strip::Geo<T>::CELLS);
    a.cblocks = ceil_div(C, strip::CH);
    const int band = y_end - y_begin;
    const long long columns = (long long)B * a.strips * a.cblocks;
    ummau::split_rows(columns, band, sms, 1, p.items, p.steps, a.seg_rows, a.segs);
    return p;
}
// Which problems go to the strips.  An image's result should not depend on the batch that it is in, so the lines see one image (all of its groups in
// SAPA-D) and lie where it is about as fast alone; batches of smaller images would gain too.  `values` of an image: channels x rows x columns.
static double values(int groups, int C, int H, int W) { return (double)groups * C * H * W; }
// at least part / whole of the columns of the strips lie inside the image
static bool strips_filled(int W, int cells, int part, int whole) { return whole * W >= part * ceil_div(W, cells) * cells; }
// The aggregation in 16 bits, us, tiles -> this one, bfloat16: 8 x 256 x 64x64 30.0 -> 17.8; one image of 64 x 64x64 6.2 -> 5.3, 32 x 32x32 4.6, 4.6, 256 x 24x24
// 4.8, 5.6 (16 of them 13.9 -> 9.8), 256 x 16x16 4.6, 5.2 (16: 9.2 -> 7.3); left with the tiles: 64 x 16x16 4.6, 4.8 (16: 6.0, 5.7).
static bool strip_pays_16(int groups, int C, int H, int W) {
    return C >= 16 && W >= 16 && (strips_filled(W, 32, 3, 4) || values(groups, C, H, W) >= 6e4);
}
// In float32, by itself (the output of av, dQ of qk, SAPA-D), its line sees the whole problem, because alone and in a batch are too far apart: 128 x 32x32 4.3,
// 5.7 here, 16 of them 18.4 -> 11.5; 64 x 64x64 5.4, 6.4, 16 of them 40.6 -> 28.1.  So these results may differ in rounding from those of the image alone.  A
// step takes about 0.75 us, whatever the channels, and four to start; the kernels on tiles 3.7 us for a million products of cells and (channels + 99).  us,
// tiles -> this one: 8 x 256 x 64x64 54 -> 37; 32 x 64 x 64x64 76 -> 51; 1 x 256 x 256x256 109 -> 77; 8 x 256 x 32x32 19 -> 14; 16 x 64 x 32x32 14.8 -> 13.5; 1 x
// 32 x 512x512 117 -> 92; and where the line leaves them with the tiles: 8 x 32 x 32x32 6.9, 9.7 here; 4 x 128 x 32x32 8.7, 8.8.
static bool strip_pays_f32(const StripPlan &p) {
    const strip::SArgs &a = p.a;
    return (double)p.steps <= 0.7 + 5.1e-6 * a.B * (a.y_end - a.y_begin) * a.W * (a.C + 99.0);
}

template <typename T>
static int launch_strip(const void *v, const void *wt, void *out, StripPlan p, int sms, cudaStream_t st) {
    using G = strip::Geo<T>;
    static const char *const name = "sapa_strip_kernel";
    strip::SArgs &a = p.a;
    const CUtensorMapDataType ty = G::F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                          : std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    constexpr int ES = (int)sizeof(T);
    CUtensorMap vmap{}, wmap{}, omap{};
    if (!make_nchw_map(&vmap, v, a.W, a.rows, a.C, a.B, strip::VROW / ES, std::min(a.C, strip::CH), 1, ty, ES, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !make_nchw_map(&wmap, wt, 2 * a.W, 2 * a.wrows, 25, a.B, G::PX, 25, 2, ty, ES, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !make_nchw_map(&omap, out, 2 * a.W, 2 * a.H, a.C, a.B, G::PX, 32, 1, ty, ES, CU_TENSOR_MAP_SWIZZLE_128B)) {
        set_error("%s: cuTensorMapEncodeTiled rejected the tensor layout", name);
        return SAPA_ERR_UNSUPPORTED;
    }
    if (p.items > 0x7fffffffLL) {
        set_error("too many tiles");
        return SAPA_ERR_ARGUMENT;
    }
    int n = 0;
    if (int e = prepare_launch(reinterpret_cast<const void *>(sapa_strip_kernel<T>), G::SMEM, name, n)) return e;
    a.v = v; a.wt = wt; a.out = out;
    launch_next(sapa_strip_kernel<T>, (unsigned)std::min<long long>(p.items, sms), strip::NT, G::SMEM, st, vmap, wmap, omap, a);
    return check_launch(name);
}

// The forward on strips takes up to 64 query channels, rows of 16 columns and more (a strip of 32 is less than half full below that) and at
// least 24 value channels, of images of twenty thousand values and more.  A channel of a large image is a page of memory of its own, and this kernel touches
// all channels of a row where the tiles touch 32 of eight rows: images of more than 100 M values in more than 64 channels stay with the tiles.  A slab
// goes the way of its image (image_rows).  bfloat16, us, tiles -> strips: 64 x 256 x 128x128 824 -> 700, 8 x 256 x 64x64 35.4 -> 27.2, 16 x 64 x 64x64 30 -> 19 (32
// query channels), 8 x 256 x 32x32 18.0 -> 11.2, 4 x 256 x 512x512 826 -> 755, 1 x 64 x 2048x1024 865 -> 777; an image alone 256 x 1024x64 64 -> 47, 64 x 64x64 8.1
// -> 6.3, 256 x 16x16 5.6, 6.0 here (16 of them 11.8 -> 10.6), 128 x 24x24 5.6, 6.6 (16: 12.1 -> 10.1); 8 columns: 64 x 256 x 16x8 19.1, 24.8; smaller images: 64 x
// 16x16 4.8, 5.2 (16: 7.0, 7.1); large ones: 1 x 256 x 1024x512 420, 458, 8192x128 865, 1014, 4096x512 1748, 2273.
static bool strip_fwd_pays(int C, int d, int W, int image_rows) {
    const double n = values(1, C, image_rows, W);
    return d <= sfwd::MAX_D && W >= 16 && C >= 24 && n >= 2e4 && (n <= 1e8 || C <= 64);
}

template <typename T>
static int launch_strip_fwd(const void *q, const void *k, const void *v, void *out, void *attn, int d, StripPlan p, int sms, cudaStream_t st) {
    static const char *const name = "sapa_strip_fwd_kernel";
    strip::SArgs &a = p.a;
    const CUtensorMapDataType ty = std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int dpad = ceil_div(d, 16) * 16;
    CUtensorMap qmap{}, kmap{}, vmap{}, omap{};
    if (!make_nchw_map(&qmap, q, 2 * a.W, 2 * a.H, d, a.B, 64, dpad, 2, ty, 2, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_nchw_map(&kmap, k, a.W, a.rows, d, a.B, 64, dpad, 1, ty, 2, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_nchw_map(&vmap, v, a.W, a.rows, a.C, a.B, strip::VROW / 2, std::min(a.C, strip::CH), 1, ty, 2, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !make_nchw_map(&omap, out, 2 * a.W, 2 * a.H, a.C, a.B, 64, 32, 1, ty, 2, CU_TENSOR_MAP_SWIZZLE_128B)) {
        set_error("%s: cuTensorMapEncodeTiled rejected the tensor layout", name);
        return SAPA_ERR_UNSUPPORTED;
    }
    if (p.items > 0x7fffffffLL) {
        set_error("too many tiles");
        return SAPA_ERR_ARGUMENT;
    }
    sfwd::FArgs f{};
    a.v = v; a.out = out;
    f.s = a; f.attn = attn; f.q = q; f.k = k; f.d = d;
    auto go = [&](auto ksteps) -> int {
        constexpr int KSTEPS = decltype(ksteps)::value, SMEM = sfwd::Lay<T, KSTEPS>::SMEM;
        int n = 0;
        if (int e = prepare_launch(reinterpret_cast<const void *>(sapa_strip_fwd_kernel<T, KSTEPS>), SMEM, name, n)) return e;
        launch_next(sapa_strip_fwd_kernel<T, KSTEPS>, (unsigned)std::min<long long>(p.items, sms), sfwd::NT, SMEM, st, qmap, kmap, vmap, omap, f);
        return check_launch(name);
    };
    return dpad == 16 ? go(std::integral_constant<int, 1>{}) : dpad == 32 ? go(std::integral_constant<int, 2>{})
           : dpad == 48 ? go(std::integral_constant<int, 3>{}) : go(std::integral_constant<int, 4>{});
}

// float32 logits of hi (d channels) and lo, their softmax, or its backward with the saved map `attn`
template <int WHAT>
static int launch_strip_sim(const void *hi, const void *lo, const void *attn, void *out, int B, int d, int H, int W, int rows, int ytop0, int y_begin, int y_end,
                            int map_rows, int map_y0, cudaStream_t st) {
    static const char *const names[3] = {"sapa_strip_sim_kernel<logits>", "sapa_strip_sim_kernel<softmax>", "sapa_strip_sim_kernel<softmax_bwd>"}, *const name = names[WHAT];
    const CUtensorMapDataType ty = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    CUtensorMap xmap{}, lmap{};
    if (!make_nchw_map(&xmap, hi, 2 * W, 2 * H, d, B, 2 * ssim::CELLS, ssim::KCH, 4, ty, 4, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !make_nchw_map(&lmap, lo, W, rows, d, B, ssim::LROW / 4, ssim::KCH, ssim::ROWS6, ty, 4, CU_TENSOR_MAP_SWIZZLE_NONE)) {
        set_error("%s: cuTensorMapEncodeTiled rejected the tensor layout", name);
        return SAPA_ERR_UNSUPPORTED;
    }
    ssim::Args a{};
    a.attn = static_cast<const float *>(attn); a.out = static_cast<float *>(out);
    a.map_rows = map_rows; a.map_y0 = map_y0;
    a.B = B; a.d = d; a.H = H; a.W = W; a.ytop0 = ytop0; a.y_begin = y_begin; a.y_end = y_end;
    a.strips = ceil_div(W, ssim::CELLS); a.pairs = ceil_div(y_end - y_begin, 2); a.stages = ceil_div(d, ssim::KCH);
    const long long units = (long long)B * a.strips * a.pairs;
    if (units > 0x7fffffffLL) {
        set_error("too many tiles");
        return SAPA_ERR_ARGUMENT;
    }
    int sms = 0;
    if (int e = prepare_launch(reinterpret_cast<const void *>(sapa_strip_sim_kernel<WHAT>), ssim::SMEM, name, sms)) return e;
    launch_next(sapa_strip_sim_kernel<WHAT>, (unsigned)std::min<long long>(units, sms), ssim::NT, ssim::SMEM, st, xmap, lmap, a);
    return check_launch(name);
}

// the same in 16 bits: logits (as float32 where asked for) or the softmax backward with the saved map `attn`
template <typename T, int WHAT>
static int launch_strip_sim_16(const void *hi, const void *lo, const void *attn, void *out, int B, int d, int H, int W, int rows, int ytop0, int y_begin, int y_end,
                               cudaStream_t st) {
    static const char *const names[3] = {"sapa_strip_sim_16_kernel<logits>", "sapa_strip_sim_16_kernel<logits_f32>", "sapa_strip_sim_16_kernel<softmax_bwd>"},
                *const name = names[WHAT];
    const CUtensorMapDataType ty = std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int kch = d <= 16 ? 16 : 32;
    CUtensorMap xmap{}, lmap{};
    if (!make_nchw_map(&xmap, hi, 2 * W, 2 * H, d, B, 2 * s16::CELLS, kch, 4, ty, 2, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_nchw_map(&lmap, lo, W, rows, d, B, 64, kch, s16::ROWS6, ty, 2, CU_TENSOR_MAP_SWIZZLE_128B)) {
        set_error("%s: cuTensorMapEncodeTiled rejected the tensor layout", name);
        return SAPA_ERR_UNSUPPORTED;
    }
    s16::Args a{};
    a.attn = attn; a.out = out;
    a.B = B; a.d = d; a.H = H; a.W = W; a.ytop0 = ytop0; a.y_begin = y_begin; a.y_end = y_end;
    a.strips = ceil_div(W, s16::CELLS); a.pairs = ceil_div(y_end - y_begin, 2); a.stages = ceil_div(d, kch);
    const long long units = (long long)B * a.strips * a.pairs;
    if (units > 0x7fffffffLL) {
        set_error("too many tiles");
        return SAPA_ERR_ARGUMENT;
    }
    auto go = [&](auto channels) -> int {
        constexpr int KCH = decltype(channels)::value, SMEM = s16::Lay<KCH>::SMEM;
        int sms = 0;
        if (int e = prepare_launch(reinterpret_cast<const void *>(sapa_strip_sim_16_kernel<T, WHAT, KCH>), SMEM, name, sms)) return e;
        launch_next(sapa_strip_sim_16_kernel<T, WHAT, KCH>, (unsigned)std::min<long long>(units, sms), s16::NT, SMEM, st, xmap, lmap, a);
        return check_launch(name);
    };
    return kch == 16 ? go(std::integral_constant<int, 16>{}) : go(std::integral_constant<int, 32>{});
}

}  // namespace tma

// K = 5, s = 2 and every row of every tensor on a 16-byte boundary; other widths take the ragged form of the kernels
bool fused_tma_supported(int W, int dtype) {
    if (tma::encode_tiled_fn() == nullptr) return false;
    if (dtype == SAPA_F32) return W % 4 == 0;
    if (dtype == SAPA_F16 || dtype == SAPA_BF16) return W % 8 == 0;
    return false;
}

int launch_fused_tma_slots(int mode, const void *q, const void *k, const void *v, void *out, void *attn, void *ws, int B, int d,
                           int C, int H, int W, int rows, int ytop0, int y_begin, int y_end, int dtype, bool slots_f32,
                           cudaStream_t st, int groups, int image_rows, void *scratch, size_t scratch_bytes);

// 16-bit: tiles of 4 x 32 instead of 4 x 8 pixels where at least three quarters of their columns are inside the image (below that
// idle warps cost what the loads save) and two thirds of the SMs get one.
// us, 4 x 8 -> 4 x 32: bfloat16 forward 8 x 256 x 64x64 55.7 -> 40.9, 64 x 256 x 128x128 1540 -> 930, 1 x 256 x 1024x1024 2520 -> 970;
// float16 forward 4 x 128 x 56x56 (112 tiles) 24.6 -> 19.4; with fewer tiles the 4 x 8 ones use more SMs: module training at
// 8 x 256 x 32x32 (64 tiles) 252 -> 264, forward of 1 x 64 x 64x64 (32 tiles) 13.2 -> 14.3.
static bool wide16_pays(int W, int tiles_y, int B) {
    const int tiles_x = ceil_div(W, tma::w16::COLS);
    return 4 * W >= 3 * tiles_x * tma::w16::COLS && (long long)B * tiles_x * tiles_y >= 100;
}

// float32 on strips of 16 columns, the similarity by itself (us, tiles -> strips: 8 images, 64 channels, 64x64 19.0 -> 14.5; 1 x 64 x 128x128 12.1 -> 8.8;
// 4 x 16 x 64x64 6.7 -> 5.0; 1 x 64 x 16x64 5.1 -> 4.4; 1 x 32 x 24x24 4.2 -> 3.7; 4 x 16 x 16x64 3.5, 3.8; left with the tiles: images of fewer than ten
// thousand values).
static bool strip_sim_pays(int groups, int C, int H, int W) {
    return tma::encode_tiled_fn() != nullptr && W % 4 == 0 && W >= 16 && tma::strips_filled(W, 16, 3, 4) && tma::values(groups, C, H, W) >= 1e4;
}
// The forward as two launches, softmax of the logits and aggregation.  An image's result depends neither on the batch it is in nor on the slab of
// rows that a process has of it (image_rows), so the line sees one image.  It gives up to two microseconds of a single image of its smallest for a
// third of a batch of them (us, tiles -> strips, 64 query channels: 128 x 64x64 12.1, 12.3 here, 4 of them 29.6 -> 21, 16 95 -> 65; with 32 query channels 10.3, 11.6, 4
// 25.5 -> 20.6; 256 x 48x48 12.1 -> 11.9; 256 x 64x64 15.6 -> 13.9; 48 x 128x128 22 -> 20; 8 x 256 x 64x64 72 -> 51) and leaves with the tiles: 64 x 64x64 10.5, 13.7 (16:
// 75, 57), 256 x 32x32 10.4, 11.1 (16: 44, 30), and flat images, 48 x 8x256 6.3, 9.7, 256 x 4x64 8.0, 9.7, 256 x 16x64 10.4, 11.0.
bool fused_f32_on_strips(int C, int W, int image_rows) {
    return tma::encode_tiled_fn() != nullptr && W % 4 == 0 && tma::strips_filled(W, 16, 3, 4) && C >= 48 && (double)W * W * C >= (C >= 96 ? 5e5 : 7.5e5) &&
           tma::values(1, C, image_rows, W) >= 3e5;
}
// Bytes of the map of one low-res row of an image; the scratch in place of the whole map, which may be half of the output's size: 256 MiB at most (as many images
// or rows as that holds at a time: 64 x 64 x 128x128, whose map has 419 MB, 614 us through one piece, 628 through two, 695 through seven of 64 MiB).
size_t fused_scratch_row(int W) { return (size_t)25 * 4 * W * sizeof(float); }
size_t fused_scratch(int B, int H, int W) {
    const size_t row = fused_scratch_row(W), limit = (size_t)256 << 20, image = row * H, all = image * B;
    return all <= limit ? all : image <= limit ? limit / image * image : std::max<size_t>(limit / row & ~(size_t)1, 2) * row;
}
// Stage 1 of the backward likewise, softmax backward of the logits and aggregation, from 64 value channels on and with four fifths of the strips' columns inside
// the image.  The line sees channels and columns alone: a slab's query gradient equals the rows of the image's.  The whole backward, us, tiles -> strips
// (gathers on tiles in both): 1 x 64 x 64x64 27.2, 27.1, 16 of them 187 -> 167; 4 x 256 x 64x64 122 -> 112, 1 x 256 x 32x32 36.7 -> 26.9, 1 x 512 x 16x16 49 -> 29;
// 24 columns, 16 x 128 x 24x24 43, 48 on strips.
static bool bwd_f32_on_strips(int C, int W) {
    return tma::encode_tiled_fn() != nullptr && W % 4 == 0 && W >= 16 && C >= 64 && tma::strips_filled(W, 16, 4, 5);
}

// 16 bits: the similarity always runs on strips (us, tiles -> strips, bfloat16: 8 images, 64 channels, 64x64 15.0 -> 11.0; 1 x 32 x 16x16 6.2 ->
// 4.3; 64 x 32 x 8x8 7.0 -> 5.4); stage 1 of the backward as two launches from 32 value channels on and with five eighths of the strips' columns inside the
// image.  The whole backward, us: 1 x 32 x 32x32 21.9, 21.5, 64 of them 89 -> 69; 1 x 256 x 64x64 33.7 -> 29.7, 16 x 64 x 64x64 105 -> 81, 4 x 256 x 24x24 32.3 ->
// 27.6, 2 x 256 x 24x40 28.8 -> 25.7; 16 columns, 64 x 256 x 64x16 239, 253 on strips.
static bool strip_bwd_16_pays(int C, int W) { return W >= 24 && C >= 32 && tma::strips_filled(W, 32, 5, 8); }

// Returns SAPA_ERR_UNSUPPORTED when a tensor map cannot be built (the caller then uses another kernel).
// mode 0 (forward): out = atn(softmax(sim(q, k)), v), attn = optional output.
// mode 1 (backward stage 1): q = grad_out [B,d,2H,2W], k = value [B,d,H,W] (d = value channels), v = key [B,C,H,W]
//        (C = key channels), attn = saved attention map (input), ws = logit gradients (output), out = grad_query.
// mode 2 (sim): attn (output) = sim(q, k); v, out unused, C ignored.   mode 3 (agg): out = atn(attn (input), v); q, k unused, d ignored.
int launch_fused_tma(int mode, const void *q, const void *k, const void *v, void *out, void *attn, void *ws, int B, int d, int C,
                     int H, int W, int rows, int ytop0, int y_begin, int y_end, int dtype, cudaStream_t st, int groups, int image_rows,
                     void *scratch, size_t scratch_bytes) {
    return launch_fused_tma_slots(mode, q, k, v, out, attn, ws, B, d, C, H, W, rows, ytop0, y_begin, y_end, dtype, false, st, groups, image_rows, scratch, scratch_bytes);
}

// slots_f32 (16-bit tensors, mode 2 only): `attn` is a float32 tensor - the logits are written at full precision while
// query and key stay 16-bit.  groups: how many of the B belong to one image (SAPA-D), image_rows: rows of the image of which a slab is a part, for the choice
// of the kernel.  scratch: in place of `attn` where the forward goes through a map (fused_scratch).
int launch_fused_tma_slots(int mode, const void *q, const void *k, const void *v, void *out, void *attn, void *ws, int B, int d,
                           int C, int H, int W, int rows, int ytop0, int y_begin, int y_end, int dtype, bool slots_f32,
                           cudaStream_t st, int groups, int image_rows, void *scratch, size_t scratch_bytes) {
    using namespace tma;
    if (slots_f32 && (dtype == SAPA_F32 || mode != MODE_SIM)) {
        set_error("sapa_tma_fused: float32 slots are for the 16-bit logit mode");
        return SAPA_ERR_UNSUPPORTED;
    }
    if (mode == MODE_SIM) C = 0;
    if (mode == MODE_AGG) d = 0;
    const bool use_qk = mode != MODE_AGG, use_v = mode != MODE_SIM;
    CUtensorMap qmap{}, kmap{}, vmap{}, omap{};
    const bool ragged = !fused_tma_supported(W, dtype);
    if (ragged && dtype == SAPA_F32) {
        set_error("sapa_tma_fused: float32 rows have to be multiples of 16 bytes");
        return SAPA_ERR_UNSUPPORTED;
    }
    const bool wide = !ragged && dtype != SAPA_F32 && wide16_pays(W, ceil_div(y_end - y_begin, ROWS), B);
    int sms = 0;
    if (!ragged)
        if (int e = device_sms("sapa_tma_fused", sms)) return e;
    auto in_type = [&](auto go) { return dtype == SAPA_F32 ? go(float{}) : dtype == SAPA_F16 ? go(__half{}) : go(__nv_bfloat16{}); };
    // the aggregation on strips, of all rows of the launch
    auto aggregate = [&](const void *wt) {
        return in_type([&](auto one) {
            using T = decltype(one);
            return launch_strip<T>(v, wt, out, strip_plan<T>(B, C, H, W, rows, ytop0, y_begin, y_end, sms), sms, st);
        });
    };
    if (mode == MODE_AGG && !ragged && (dtype == SAPA_F32 ? strip_pays_f32(strip_plan<float>(B, C, H, W, rows, ytop0, y_begin, y_end, sms)) : strip_pays_16(groups, C, H, W)))
        return aggregate(attn);
    if (dtype == SAPA_F32 && mode == MODE_FWD && (attn != nullptr || scratch_bytes > 0) && fused_f32_on_strips(C, W, image_rows)) {
        // images n0 .., rows y0 .. y1 - 1 through a map that holds low-res rows map_y0 and on of each image
        auto part = [&](int n0, int images, int y0, int y1, void *map, int map_rows, int map_y0) -> int {
            const size_t hi = (size_t)(2 * H) * (2 * W), lo = (size_t)rows * W;
            const float *qn = static_cast<const float *>(q) + (size_t)n0 * d * hi, *kn = static_cast<const float *>(k) + (size_t)n0 * d * lo, *vn = static_cast<const float *>(v) + (size_t)n0 * C * lo;
            if (int e = launch_strip_sim<ssim::SOFTMAX>(qn, kn, nullptr, map, images, d, H, W, rows, ytop0, y0, y1, map_rows, map_y0, st)) return e;
            StripPlan p = strip_plan<float>(images, C, H, W, rows, ytop0, y0, y1, sms);
            p.a.wrows = map_rows; p.a.wy0 = map_y0;
            return launch_strip<float>(vn, map, static_cast<float *>(out) + (size_t)n0 * C * hi, p, sms, st);
        };
        if (attn != nullptr) return part(0, B, y_begin, y_end, attn, H, 0);
        // scratch: as many images at a time as it holds the rows of, or bands of rows of an image
        const size_t row_bytes = fused_scratch_row(W), band = (size_t)(y_end - y_begin);
        const int images = (int)std::min<size_t>((size_t)B, scratch_bytes / (row_bytes * band));
        const int step = images > 0 ? (int)band : (int)(scratch_bytes / row_bytes) & ~1;
        for (int n0 = 0; n0 < B; n0 += std::max(images, 1))
            for (int y0 = y_begin; y0 < y_end; y0 += step)
                if (int e = part(n0, std::min(std::max(images, 1), B - n0), y0, std::min(y0 + step, y_end), scratch, std::min(step, y_end - y0), y0)) return e;
        return SAPA_OK;
    }
    if (dtype == SAPA_F32 && mode == MODE_SIM && strip_sim_pays(groups, d, H, W))
        return launch_strip_sim<ssim::LOGITS>(q, k, nullptr, attn, B, d, H, W, rows, ytop0, y_begin, y_end, H, 0, st);
    if (dtype == SAPA_F32 && mode == MODE_BWD && bwd_f32_on_strips(d, W)) {
        const int e = launch_strip_sim<ssim::SOFTMAX_BWD>(q, k, attn, ws, B, d, H, W, rows, ytop0, y_begin, y_end, H, 0, st);
        return e != SAPA_OK ? e : aggregate(ws);
    }
    if (dtype != SAPA_F32 && !ragged && (mode == MODE_SIM || (mode == MODE_BWD && strip_bwd_16_pays(d, W)))) {
        auto go = [&](auto one) -> int {
            using T = decltype(one);
            return mode == MODE_BWD ? launch_strip_sim_16<T, s16::SOFTMAX_BWD>(q, k, attn, ws, B, d, H, W, rows, ytop0, y_begin, y_end, st)
                   : slots_f32      ? launch_strip_sim_16<T, s16::LOGITS_F32>(q, k, nullptr, attn, B, d, H, W, rows, ytop0, y_begin, y_end, st)
                                    : launch_strip_sim_16<T, s16::LOGITS>(q, k, nullptr, attn, B, d, H, W, rows, ytop0, y_begin, y_end, st);
        };
        const int e = dtype == SAPA_F16 ? go(__half{}) : go(__nv_bfloat16{});
        return e != SAPA_OK || mode == MODE_SIM ? e : aggregate(ws);
    }
    if (mode == MODE_FWD && !ragged && dtype != SAPA_F32 && strip_fwd_pays(C, d, W, image_rows)) {
        auto go = [&](auto one) -> int {
            using T = decltype(one);
            return launch_strip_fwd<T>(q, k, v, out, attn, d, strip_plan<T>(B, C, H, W, rows, ytop0, y_begin, y_end, sms), sms, st);
        };
        return dtype == SAPA_F16 ? go(__half{}) : go(__nv_bfloat16{});
    }
    bool ok = true;
    if (ragged) {
    } else if (dtype == SAPA_F32) {
        const auto ty = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
        const auto sw = CU_TENSOR_MAP_SWIZZLE_64B;
        if (use_qk) ok = ok && make_nchw_map(&qmap, q, 2 * W, 2 * H, d, B, HC, F_KCH, HH, ty, 4, sw) && make_nchw_map(&kmap, k, W, rows, d, B, HC, F_KCH, HH, ty, 4, sw);
        if (use_v) ok = ok && make_nchw_map(&vmap, v, W, rows, C, B, HC, F_VCH, HH, ty, 4, sw) && make_nchw_map(&omap, out, 2 * W, 2 * H, C, B, HC, F_VCH, HH, ty, 4, sw);
    } else if (wide) {
        const auto ty = dtype == SAPA_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
        if (use_qk) ok = ok && make_nchw_map(&qmap, q, 2 * W, 2 * H, d, B, w16::BC, w16::KCH, HH, ty, 2, sw) && make_nchw_map(&kmap, k, W, rows, d, B, w16::BC, w16::KCH, HH, ty, 2, sw);
        if (use_v) ok = ok && make_nchw_map(&vmap, v, W, rows, C, B, w16::BC, w16::VCH, HH, ty, 2, sw) &&
                        make_nchw_map(&omap, out, 2 * W, 2 * H, C, B, 2 * w16::COLS, w16::VCH, 2, ty, 2, sw);
    } else {
        const auto ty = dtype == SAPA_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        if (use_qk) ok = ok && make_nchw_map(&qmap, q, 2 * W, 2 * H, d, B, 16, h16::KCH, HH, ty, 2, CU_TENSOR_MAP_SWIZZLE_32B) &&
                         make_nchw_map(&kmap, k, W, rows, d, B, h16::BC, h16::KCH, HH, ty, 2, CU_TENSOR_MAP_SWIZZLE_NONE);
        if (use_v) ok = ok && make_nchw_map(&vmap, v, W, rows, C, B, h16::BC, h16::VCH, HH, ty, 2, CU_TENSOR_MAP_SWIZZLE_NONE);
    }
    if (!ok) {
        set_error("sapa_tma_fused (mode %d): cuTensorMapEncodeTiled rejected the tensor layout (CUresult %d)", mode,
                  last_encode_result());
        return SAPA_ERR_UNSUPPORTED;
    }
    // maps a mode never touches still travel as kernel parameters: give them defined contents
    if (!use_qk) { qmap = vmap; kmap = vmap; }
    if (!use_v) { vmap = kmap; omap = kmap; }
    if (dtype != SAPA_F32 && !(wide && use_v)) omap = vmap;
    Args a{};
    a.q = q; a.k = k; a.v = v;
    a.out = out; a.attn = attn; a.ws = ws;
    a.B = B; a.d = d; a.C = C; a.H = H; a.W = W; a.rows = rows; a.ytop0 = ytop0;
    static_assert(F_VCH == h16::VCH, "both kernels take the same number of value channels per stage");
    a.csplit = 1; a.vstages = ceil_div(C, F_VCH);
    static_assert(h16::COLS == COLS, "both kernels use the same tile");
    a.y_begin = y_begin; a.y_end = y_end;
    a.tiles_x = ceil_div(W, wide ? w16::COLS : COLS);
    a.tiles_y = ceil_div(y_end - y_begin, ROWS);
    constexpr int smem32 = NSTAGE * SLOT_BYTES + 2 * O_BYTES + 1024;
    static const char *const names32[4] = {"sapa_tma_fused_f32_kernel<fwd>", "sapa_tma_fused_f32_kernel<bwd>",
                                           "sapa_tma_fused_f32_kernel<sim>", "sapa_tma_fused_f32_kernel<agg>"};
    static const char *const names16[4] = {"sapa_tma_fused_16_kernel<fwd>", "sapa_tma_fused_16_kernel<bwd>",
                                           "sapa_tma_fused_16_kernel<sim>", "sapa_tma_fused_16_kernel<agg>"};
    static const char *const names_wide[4] = {"sapa_wide_16_kernel<fwd>", "sapa_wide_16_kernel<bwd>", "sapa_wide_16_kernel<sim>", "sapa_wide_16_kernel<agg>"};
    static const char *const names_ragged[4] = {"sapa_tma_fused_16_kernel<ragged fwd>", "sapa_tma_fused_16_kernel<ragged bwd>",
                                                "sapa_tma_fused_16_kernel<ragged sim>", "sapa_tma_fused_16_kernel<ragged agg>"};
#define SAPA_TMA_LAUNCH32(M)                                                                                                             \
    case M:                                                                                                                              \
        return launch_persistent(sapa_tma_fused_f32_kernel<M>, names32[M], NT, smem32, CTAS_PER_SM, M != MODE_BWD, a, st, qmap, kmap, vmap, omap);
#define SAPA_TMA_LAUNCH16(T, M)                                                                                                          \
    case M:                                                                                                                              \
        return ragged ? launch_persistent(sapa_tma_fused_16_kernel<T, M, true>, names_ragged[M], h16::NT_RAGGED, h16::SMEM_BYTES, 1, M != MODE_BWD, a, st, qmap, kmap, vmap) \
               : wide ? launch_persistent(sapa_wide_16_kernel<T, M>, names_wide[M], w16::NT, w16::SMEM_BYTES, 1, false, a, st, qmap, kmap, vmap, omap) \
                      : launch_persistent(sapa_tma_fused_16_kernel<T, M, false>, names16[M], h16::NT, h16::SMEM_BYTES, h16::CTAS_PER_SM, M != MODE_BWD, a, st, qmap, kmap, vmap);
#define SAPA_TMA_LAUNCH16_SIM(T)         /* ragged rows: the others have gone to the strips */                                           \
    case MODE_SIM:                                                                                                                       \
        return launch_persistent(sapa_tma_fused_16_kernel<T, MODE_SIM, true>, names_ragged[MODE_SIM], h16::NT_RAGGED, h16::SMEM_BYTES, 1, true, a, st, qmap, kmap, vmap);
    if (dtype == SAPA_F32) switch (mode) { SAPA_TMA_LAUNCH32(MODE_FWD) SAPA_TMA_LAUNCH32(MODE_BWD) SAPA_TMA_LAUNCH32(MODE_SIM) SAPA_TMA_LAUNCH32(MODE_AGG) }
    if (dtype == SAPA_F16)
        switch (mode) { SAPA_TMA_LAUNCH16(__half, MODE_FWD) SAPA_TMA_LAUNCH16(__half, MODE_BWD) SAPA_TMA_LAUNCH16_SIM(__half) SAPA_TMA_LAUNCH16(__half, MODE_AGG) }
    if (dtype == SAPA_BF16)
        switch (mode) { SAPA_TMA_LAUNCH16(__nv_bfloat16, MODE_FWD) SAPA_TMA_LAUNCH16(__nv_bfloat16, MODE_BWD) SAPA_TMA_LAUNCH16_SIM(__nv_bfloat16) SAPA_TMA_LAUNCH16(__nv_bfloat16, MODE_AGG) }
    set_error("sapa_tma_fused: unknown mode %d or dtype code %d", mode, dtype);
    return SAPA_ERR_ARGUMENT;
#undef SAPA_TMA_LAUNCH32
#undef SAPA_TMA_LAUNCH16
#undef SAPA_TMA_LAUNCH16_SIM
}

// One CTA waits, with a short limit, on a shared-memory barrier that nothing ever signals: the bounded wait gives up,
// the kernel raises g_wait_timeout exactly as the production kernels would and returns normally.
__global__ void sapa_wait_selftest_kernel(int tries) {
    __shared__ __align__(8) unsigned long long bars[4];
    const unsigned addr = (unsigned)__cvta_generic_to_shared(bars), ring = addr + 8;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i) tmau::mbar_init(addr + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        bool done = false;
        for (int i = 0; i < tries && !done; ++i) done = tmau::mbar_try_wait(addr, 0);
        // what a producer does then, at two positions of a ring of three stages: one stage issued and landed, then four
        tmau::mbar_arrive(ring);
        bool landed = tmau::drain_loads<3>(ring, 1, 0);
        for (int i = 1; i <= 3; ++i) tmau::mbar_arrive(ring + 8 * (i % 3));
        landed = tmau::drain_loads<3>(ring, 1, 1) && landed;
        if (!done && landed) atomicExch(&tma::g_wait_timeout, 1);
    }
}

int launch_wait_selftest(cudaStream_t st) {
    sapa_wait_selftest_kernel<<<1, 32, 0, st>>>(64);
    return check_launch("sapa_wait_selftest_kernel");
}

// 1 if a bounded mbarrier wait of the TMA kernels gave up on the current device since the last query (synchronises the
// device).  A CTA that gives up leaves without taking part in the last-CTA reset of its scheduler pair, so a raised
// flag also means that pair may be dirty: reading a raised flag clears it and zeroes every scheduler pair.
int tma_wait_timeout_flag() {
    int flag = 0;
    if (cudaMemcpyFromSymbol(&flag, tma::g_wait_timeout, sizeof(int)) != cudaSuccess) return -1;
    if (flag != 0) {
        static const unsigned zeros[tmau::SCHED_SLOTS] = {};
        const int zero = 0;
        if (cudaMemcpyToSymbol(tma::g_next_tile, zeros, sizeof(zeros)) != cudaSuccess ||
            cudaMemcpyToSymbol(tma::g_ctas_done, zeros, sizeof(zeros)) != cudaSuccess ||
            cudaMemcpyToSymbol(tma::g_wait_timeout, &zero, sizeof(int)) != cudaSuccess)
            return -1;
    }
    return flag;
}

}  // namespace sapa
