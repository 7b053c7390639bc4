// sapa_wide16.cuh — the 16-bit kernel of sapa_tma.cu on tiles of 4 x 32 low-res pixels (8 x 64 high-res), for images wide enough to
// fill them.  Included by sapa_tma.cu, inside namespace sapa::tma.
//
// What it changes against the 4 x 8 tiles, whose time was the sum of its loads (27 us at B=8, C=256, d=64, 64x64 -> 128x128: the
// tensor memory accelerator needs two clocks for a 48-byte row as for a 128-byte one), its fragment loads and its stores:
//   * boxes are 64 columns wide (128-byte rows, 128-byte swizzle, from x0 - 16: a 32-byte boundary), so a row of loads serves
//     four times as many pixels and touches a page of a large plane a quarter as often;
//   * outputs go through shared memory and leave as boxes with rows of 128 bytes (one lane of a spare warp issues them): a store
//     from registers writes eight channels, 32 bytes each, which costs the load / store unit eight cycles (it was 70 % busy, and
//     what the kernel waited for) and an address translation per channel: 64 x 256 x 128x128 1058 -> 829 us, 1 x 256 x 1024x1024,
//     whose channels are 8 MB apart, 1666 -> 854 (in runs of a few launches; back to back 930 and 960);
//   * a warp owns 8 low-res columns of one low-res row and BOTH of its high-res rows: a key or value fragment is loaded once for
//     four products instead of twice for two each.
// Fragments, accumulation order and roundings are those of the 4 x 8 kernel (the 24 columns that a warp reads are the same
// relative to its pixels), so results are bit-identical.
namespace w16 {
constexpr int COLS = 32;                        // low-res columns of a CTA tile
constexpr int NW = ROWS * (COLS / 8);           // 16 consumer warps: (low-res row, 8 columns)
constexpr int NT = (NW + 4) * 32;               // + a warpgroup of which one lane produces: the other registers of its share go
                                                // to the consumers (16 x 112 + 4 x 24 of the 20 x 96 that the block is launched with)
constexpr int KCH = 16;                         // key / query channels per stage
constexpr int VCH = 32;                         // value channels per stage
constexpr int BC = 64;                          // box columns: x0 - 16 .. x0 + 47
constexpr int ROWB = BC * 2;                    // 128 bytes: a key / value row, and 64 high-res pixels of a query row
constexpr int K_BYTES = HH * KCH * ROWB;        // 16 KB
constexpr int Q_BYTES = 2 * ROWS * KCH * ROWB;  // 16 KB
constexpr int V_BYTES = HH * VCH * ROWB;        // 32 KB
constexpr int SLOT_BYTES = V_BYTES;
constexpr int NSTAGE = 5;
constexpr int O_BYTES = 2 * ROWS * VCH * ROWB;  // 32 KB: output box [8 high-res rows][32 channels][64 pixels], two of them behind the ring
constexpr int SMEM_BYTES = NSTAGE * SLOT_BYTES + 2 * O_BYTES + 1024;
static_assert(K_BYTES + Q_BYTES <= SLOT_BYTES && SMEM_BYTES <= 227 * 1024, "ring");
}  // namespace w16

template <typename T, int MODE>
__global__ void __launch_bounds__(w16::NT, 1)
sapa_wide_16_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                    const __grid_constant__ CUtensorMap omap, const Args a) {
    using namespace w16;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * w16::NSTAGE + 4];  // full[NSTAGE], empty[NSTAGE]; written[2], free[2] of the output boxes
    __shared__ int tile_ids[8];       // tile_ids[ti & 7] = item of the ti-th turn of this CTA, -1 = no more (the producer is at most NSTAGE turns ahead)
    const unsigned ring_addr = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned full_addr = (unsigned)__cvta_generic_to_shared(bars), empty_addr = full_addr + 8 * w16::NSTAGE;
    const unsigned written_addr = empty_addr + 8 * w16::NSTAGE, free_addr = written_addr + 16, obuf_addr = ring_addr + w16::NSTAGE * w16::SLOT_BYTES;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wrow = warp & 3, wcol = warp >> 2;
    const int g = lane >> 2, t = lane & 3;
    const int sW = 2 * a.W;
    const size_t hi_plane = (size_t)(2 * a.H) * sW;
    const int nk = (a.d + w16::KCH - 1) / w16::KCH, nv = a.vstages, total = nk + nv;
    // csplit is 1 here (at least 100 tiles); the kernel compiled without it was slower: 64 x 256 x 128x128 826 -> 840 us
    const int nitems = a.B * a.tiles_x * a.tiles_y * a.csplit;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < w16::NSTAGE; ++i) {
            mbar_init(full_addr + 8 * i, 1);
            mbar_init(empty_addr + 8 * i, w16::NW);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mbar_init(written_addr + 8 * i, w16::NW);
            mbar_init(free_addr + 8 * i, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    begin_after_previous();

    if (warp >= w16::NW) {            // producer: one lane; the stages of successive items form one stream through the ring
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;\n");
        if (tid == (w16::NW + 1) * 32) {
            // output: one lane of another warp of the group stores the boxes that the consumers have written
            int buf = 0, par = 0;
            for (int ti = 0;; ++ti) {
                for (int it = 0; it < nv; ++it) {
                    const bool ok = mbar_wait_bounded(written_addr + 8 * buf, par);
                    if (!ok) atomicExch(&g_wait_timeout, 1);
                    int u = ok ? tile_ids[ti & 7] : -1;     // as the consumers read it, at most two stages ago
                    if (u < 0) {
                        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
                        return;
                    }
                    const int c0 = (u % a.csplit * nv + it) * w16::VCH; u /= a.csplit;
                    const int x0 = (u % a.tiles_x) * w16::COLS; u /= a.tiles_x;
                    const int y0 = a.y_begin + (u % a.tiles_y) * ROWS, n = u / a.tiles_y;
                    for (int row = 0; row < ROWS && y0 + row < a.y_end; ++row)       // pixels and channels beyond the tensor are cut off
                        tma_store_4d(&omap, obuf_addr + buf * w16::O_BYTES + row * (w16::O_BYTES / ROWS), 2 * x0, c0, 2 * (y0 + row), n);
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                    asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                    mbar_arrive(free_addr + 8 * buf);
                    if (++buf == 2) { buf = 0; par ^= 1; }
                }
            }
        }
        if (tid != w16::NW * 32) return;
        int slot = 0, phase = 0;
        for (int ti = 0;; ++ti) {
            int item = (int)blockIdx.x;
            if (ti > 0) item = (int)(atomicAdd(&g_next_tile[a.sched_slot], 1u) + gridDim.x);
            if (item >= nitems) item = -1;
            int x0 = 0, y0 = 0, n = 0, vb = 0;
            if (item >= 0) {
                int u = item;
                vb = u % a.csplit * nv; u /= a.csplit;
                x0 = (u % a.tiles_x) * w16::COLS; u /= a.tiles_x;
                y0 = a.y_begin + (u % a.tiles_y) * ROWS; n = u / a.tiles_y;
            }
            for (int it = 0; it < (item < 0 ? 1 : total); ++it) {
                if (!mbar_wait_bounded(empty_addr + 8 * slot, phase ^ 1)) {
                    atomicExch(&g_wait_timeout, 1);
                    drain_loads<w16::NSTAGE>(full_addr, slot, phase);
                    return;
                }
                const unsigned bar = full_addr + 8 * slot, dst = ring_addr + slot * w16::SLOT_BYTES;
                if (it == 0) tile_ids[ti & 7] = item;
                if (item < 0) {
                    mbar_arrive(bar);          // completes the phase without data: the warps read -1 and stop
                } else if (it < nk) {
                    mbar_expect_tx(bar, w16::K_BYTES + w16::Q_BYTES);
                    tma_load_4d(dst, &kmap, bar, x0 - 16, it * w16::KCH, a.ytop0 + y0 - 2, n);
                    tma_load_4d(dst + w16::K_BYTES, &qmap, bar, 2 * x0, it * w16::KCH, 2 * y0, n);
                } else {
                    mbar_expect_tx(bar, w16::V_BYTES);
                    tma_load_4d(dst, &vmap, bar, x0 - 16, (vb + it - nk) * w16::VCH, a.ytop0 + y0 - 2, n);
                }
                if (++slot == w16::NSTAGE) { slot = 0; phase ^= 1; }
            }
            if (item < 0) {
                if (atomicAdd(&g_ctas_done[a.sched_slot], 1u) == gridDim.x - 1) {   // last CTA out: reset the scheduler slot
                    g_next_tile[a.sched_slot] = 0u;
                    g_ctas_done[a.sched_slot] = 0u;
                }
                return;
            }
        }
    }

    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;\n");

    // ---- per-lane fragment addresses (see the 4 x 8 kernel): the warp reads the 16-byte chunks wcol + 1 .. wcol + 3 of a key /
    // value row and 2 wcol, 2 wcol + 1 of a query row; a chunk's place is its index XOR (channel & 7)
    const int row_a = (lane & 7) + 8 * ((lane >> 3) & 1), chunk_a = lane >> 4, row_t = (lane & 7) + 8 * (lane >> 4), chunk_t = (lane >> 3) & 1, sw = lane & 7;
    const int q_off = w16::K_BYTES + 2 * wrow * (w16::KCH * w16::ROWB) + row_a * w16::ROWB + (((2 * wcol + chunk_a) ^ sw) << 4);
    const int k_off = wrow * (w16::KCH * w16::ROWB) + row_t * w16::ROWB + (((wcol + 1 + chunk_t) ^ sw) << 4);
    const int k_off2 = wrow * (w16::KCH * w16::ROWB) + row_a * w16::ROWB + (((wcol + 3) ^ sw) << 4);
    const int v_off = wrow * (w16::VCH * w16::ROWB) + row_a * w16::ROWB + (((wcol + 1 + chunk_a) ^ sw) << 4);
    const int o_off = 2 * wrow * (w16::VCH * w16::ROWB) + g * w16::ROWB + (((2 * wcol) ^ g) << 4) + 4 * t;      // output: chunk 2 wcol, the right group's is that ^ 1
    const int v_off2 = wrow * (w16::VCH * w16::ROWB) + row_a * w16::ROWB + (((wcol + 3) ^ sw) << 4);
    bool ok_lo[2], ok_hi[2];
    int dx_lo[2];                 // window column of the lo cell (hi = lo + 8)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        dx_lo[p] = 4 * p + g - t - 6;
        ok_lo[p] = dx_lo[p] >= 0 && dx_lo[p] <= 4;
        ok_hi[p] = dx_lo[p] + 8 >= 0 && dx_lo[p] + 8 <= 4;
    }

    const size_t plane_w = hi_plane >> 1;         // strides in 32-bit words (two elements)
    const int row_w = sW >> 1;
    constexpr float LOG2E = 1.4426950408889634f;
    int slot = 0, phase = 0, obuf = 0, opar = 0;
    for (int ti = 0;; ++ti) {
        if (!mbar_wait_bounded(full_addr + 8 * slot, phase)) { atomicExch(&g_wait_timeout, 1); return; }
        int item = tile_ids[ti & 7];              // published by the producer before the barrier's phase completed
        if (item < 0) {
            // the storing lane reads -1 and stops
            if (!mbar_wait_bounded(free_addr + 8 * obuf, opar ^ 1)) atomicExch(&g_wait_timeout, 1);
            else if (lane == 0) mbar_arrive(written_addr + 8 * obuf);
            break;
        }
        int c0 = item % a.csplit * nv * w16::VCH; item /= a.csplit;
        const int x0 = (item % a.tiles_x) * w16::COLS + 8 * wcol; item /= a.tiles_x;      // first column of this warp
        const int y = a.y_begin + (item % a.tiles_y) * ROWS + wrow, n = item / a.tiles_y;
        // rows of length 8k: the warp's columns are inside the image together or not at all
        const bool live = y < a.y_end && x0 < a.W;
        // this lane's first word of the slot tensors / the output: pixels 2t, 2t + 1 of the left group in the upper high-res row
        const size_t pix_w = (((size_t)(2 * y) * sW) >> 1) + x0 + t;

        unsigned pb[2][2][5][2];                  // [group][high-res row][dy][lo, hi]: B fragments of the aggregation
        const auto load_slots = [&](const unsigned *ap, int p, int r, int dy, unsigned &lo, unsigned &hi) {
            lo = hi = 0u;
            if (live && ok_lo[p]) lo = ap[(size_t)(dy * 5 + dx_lo[p]) * plane_w + r * row_w + 4 * p];
            if (live && ok_hi[p]) hi = ap[(size_t)(dy * 5 + dx_lo[p] + 8) * plane_w + r * row_w + 4 * p];
        };
        if (MODE == MODE_AGG) {                   // the weights come from memory, already in the packed pair layout
            const unsigned *ap = static_cast<const unsigned *>(a.attn) + (size_t)n * 25 * plane_w + pix_w;
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) load_slots(ap, p, r, dy, pb[p][r][dy][0], pb[p][r][dy][1]);
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        pb[p][r][dy][0] = movmatrix_trans(pb[p][r][dy][0]);
                        pb[p][r][dy][1] = movmatrix_trans(pb[p][r][dy][1]);
                    }
        }
        if (MODE != MODE_AGG) {
            // ------------------------------------------------------------- logits
            float s[2][2][5][4];                  // [group][high-res row][dy][(lo,px0) (lo,px1) (hi,px0) (hi,px1)]
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                        for (int i = 0; i < 4; ++i) s[p][r][dy][i] = 0.f;
            for (int it = 0; it < nk; ++it) {
                if (it > 0 && !mbar_wait_bounded(full_addr + 8 * slot, phase)) { atomicExch(&g_wait_timeout, 1); return; }
                const unsigned stage = ring_addr + slot * w16::SLOT_BYTES;
                if (live) {
                    unsigned qb[2][4];
                    ldsm_x4_trans(qb[0], stage + q_off);
                    ldsm_x4_trans(qb[1], stage + q_off + w16::KCH * w16::ROWB);
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {
                        unsigned ka[4], kc[2];
                        ldsm_x4_trans(ka, stage + k_off + dy * (w16::KCH * w16::ROWB));
                        ldsm_x2_trans(kc, stage + k_off2 + dy * (w16::KCH * w16::ROWB));
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            mma_h16<T>(s[0][r][dy], ka[0], ka[1], ka[2], ka[3], qb[r][0], qb[r][1]);
                            mma_h16<T>(s[1][r][dy], ka[1], kc[0], ka[3], kc[1], qb[r][2], qb[r][3]);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_addr + 8 * slot);
                if (++slot == w16::NSTAGE) { slot = 0; phase ^= 1; }
            }
            // ------------------------------------------------------------- between the phases, one high-res row of a group at a time
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float (&sp)[5][4] = s[p][r];
                    unsigned (&pp)[5][2] = pb[p][r];
                    const size_t at_w = (size_t)n * 25 * plane_w + pix_w + r * row_w + 4 * p;
                    if (MODE == MODE_BWD) {
                        // softmax backward; the saved attention map is read and the logit gradients are written as pairs
                        const unsigned *ap = static_cast<const unsigned *>(a.attn) + (size_t)n * 25 * plane_w + pix_w;
                        unsigned *wp = static_cast<unsigned *>(a.ws) + at_w;
                        unsigned raw[5][2];
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) load_slots(ap, p, r, dy, raw[dy][0], raw[dy][1]);
                        float d0 = 0.f, d1 = 0.f;
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            const float2 flo = unpack_pair(T(), raw[dy][0]), fhi = unpack_pair(T(), raw[dy][1]);
                            d0 += flo.x * sp[dy][0] + fhi.x * sp[dy][2];
                            d1 += flo.y * sp[dy][1] + fhi.y * sp[dy][3];
                        }
#pragma unroll
                        for (int sh = 4; sh < 32; sh <<= 1) {
                            d0 += __shfl_xor_sync(0xffffffffu, d0, sh);
                            d1 += __shfl_xor_sync(0xffffffffu, d1, sh);
                        }
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            const float2 flo = unpack_pair(T(), raw[dy][0]), fhi = unpack_pair(T(), raw[dy][1]);
                            pp[dy][0] = pack_pair(T(), flo.x * (sp[dy][0] - d0), flo.y * (sp[dy][1] - d1));
                            pp[dy][1] = pack_pair(T(), fhi.x * (sp[dy][2] - d0), fhi.y * (sp[dy][3] - d1));
                            if (live && ok_lo[p]) wp[(size_t)(dy * 5 + dx_lo[p]) * plane_w] = pp[dy][0];
                            if (live && ok_hi[p]) wp[(size_t)(dy * 5 + dx_lo[p] + 8) * plane_w] = pp[dy][1];
                        }
                    }
                    if (MODE == MODE_FWD) {
                        // softmax over the 25 window slots of each pixel: 5 rows here x the lanes with the same t.
                        // exp(x - m) = 2^(x * log2(e) - m * log2(e)): one FMA and one ex2 per element.
                        float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            if (ok_lo[p]) { m0 = fmaxf(m0, sp[dy][0]); m1 = fmaxf(m1, sp[dy][1]); }
                            if (ok_hi[p]) { m0 = fmaxf(m0, sp[dy][2]); m1 = fmaxf(m1, sp[dy][3]); }
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
                            sp[dy][0] = ok_lo[p] ? ex2_ftz(fmaf(sp[dy][0], LOG2E, -m0)) : 0.f;
                            sp[dy][1] = ok_lo[p] ? ex2_ftz(fmaf(sp[dy][1], LOG2E, -m1)) : 0.f;
                            sp[dy][2] = ok_hi[p] ? ex2_ftz(fmaf(sp[dy][2], LOG2E, -m0)) : 0.f;
                            sp[dy][3] = ok_hi[p] ? ex2_ftz(fmaf(sp[dy][3], LOG2E, -m1)) : 0.f;
                            z0 += sp[dy][0] + sp[dy][2];
                            z1 += sp[dy][1] + sp[dy][3];
                        }
#pragma unroll
                        for (int sh = 4; sh < 32; sh <<= 1) {
                            z0 += __shfl_xor_sync(0xffffffffu, z0, sh);
                            z1 += __shfl_xor_sync(0xffffffffu, z1, sh);
                        }
                        const float i0 = __frcp_rn(z0), i1 = __frcp_rn(z1);
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            pp[dy][0] = pack_pair(T(), sp[dy][0] * i0, sp[dy][1] * i1);
                            pp[dy][1] = pack_pair(T(), sp[dy][2] * i0, sp[dy][3] * i1);
                        }
                    }
                    if (MODE == MODE_FWD && a.attn != nullptr && c0 == 0 && live) {
                        unsigned *an = static_cast<unsigned *>(a.attn) + at_w;
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            if (ok_lo[p]) an[(size_t)(dy * 5 + dx_lo[p]) * plane_w] = pp[dy][0];
                            if (ok_hi[p]) an[(size_t)(dy * 5 + dx_lo[p] + 8) * plane_w] = pp[dy][1];
                        }
                    }
#pragma unroll
                    for (int dy = 0; dy < 5; ++dy) {  // S^T accumulator fragments -> B fragments of the aggregation
                        pp[dy][0] = movmatrix_trans(pp[dy][0]);
                        pp[dy][1] = movmatrix_trans(pp[dy][1]);
                    }
                }
        }
        // ------------------------------------------------------------- aggregation
        for (int it = 0; it < nv; ++it) {
            if ((MODE != MODE_AGG || it > 0) && !mbar_wait_bounded(full_addr + 8 * slot, phase)) { atomicExch(&g_wait_timeout, 1); return; }
            const unsigned stage = ring_addr + slot * w16::SLOT_BYTES;
            float acc[2][2][2][4];                // [16 channels][high-res row][group]
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int p = 0; p < 2; ++p)
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[b][r][p][i] = 0.f;
            if (live) {
#pragma unroll
                for (int dy = 0; dy < 5; ++dy)
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        unsigned va[4], vc[2];
                        ldsm_x4(va, stage + v_off + dy * (w16::VCH * w16::ROWB) + b * 16 * w16::ROWB);
                        ldsm_x2(vc, stage + v_off2 + dy * (w16::VCH * w16::ROWB) + b * 16 * w16::ROWB);
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            mma_h16<T>(acc[b][r][0], va[0], va[1], va[2], va[3], pb[0][r][dy][0], pb[0][r][dy][1]);
                            mma_h16<T>(acc[b][r][1], va[2], va[3], vc[0], vc[1], pb[1][r][dy][0], pb[1][r][dy][1]);
                        }
                    }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_addr + 8 * slot);
            if (++slot == w16::NSTAGE) { slot = 0; phase ^= 1; }
            // D fragments -> output box, 128-byte swizzle: the 32 lanes of a store hit 32 banks
            if (!mbar_wait_bounded(free_addr + 8 * obuf, opar ^ 1)) { atomicExch(&g_wait_timeout, 1); return; }
            const unsigned ob = obuf_addr + obuf * w16::O_BYTES + o_off;
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int j = 0; j < w16::VCH / 8; ++j)         // channel g + 8j: block j/2, half j%2
                        sts32((ob ^ (p << 4)) + r * (w16::VCH * w16::ROWB) + 8 * j * w16::ROWB,
                              pack_pair(T(), acc[j >> 1][r][p][2 * (j & 1)], acc[j >> 1][r][p][2 * (j & 1) + 1]));
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(written_addr + 8 * obuf);
            if (++obuf == 2) { obuf = 0; opar ^= 1; }
        }
    }
}
