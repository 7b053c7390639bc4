// sapa_gath_wide16.cuh — the 16-bit gather on tiles of 4 x 32 output cells, for images wide enough to fill them.  Included by
// sapa_gath_mma.cu, inside namespace sapa::gmma.
//
// What it changes against the 4 x 8 tiles, whose boxes are four times the pixels of their cells in 64-byte rows and whose
// fragments take two shared-memory loads for one m16n8k8:
//   * a box row holds the 80 pixels that 32 columns reach (64 in rows of 128 bytes, 128-byte swizzle, from pixel 2 * x0 - 8, and 16
//     in rows of 32 bytes, 32-byte swizzle): 1.25 times the pixels instead of twice;
//   * a warp owns 8 columns of one output row with BOTH high-res rows of their parents: the k dimension of an m16n8k16 is 8 pixels
//     of the upper and the same 8 of the lower row, A comes from one ldmatrix.x4 (16 channels x those 16 pixels), and no partial
//     sums pass between warps.
// It is bound by the shared-memory reads of the fragments (1280 clocks a stage on paper, the MMAs 700).  bfloat16, value gradient of
// 8 x 256 x 64x64: 62 -> 29 us alone; 32 groups of 64 channels: 80 -> 49 us.
namespace gw16 {
constexpr int COLS = 32;
constexpr int NW = ROWS * (COLS / 8);            // 16 consumer warps: (output row, 8 columns)
constexpr int NT = (NW + 4) * 32;                // + a warpgroup of which one lane produces: the other registers of its share go
                                                 // to the consumers (16 x 112 + 4 x 24 of the 20 x 96 that the block is launched with)
constexpr int NCH = 16;                          // channels per stage
constexpr int ROW_A = 128, ROW_B = 32;           // bytes of a box row: 64 and 16 pixels
constexpr int A_BYTES = HR * NCH * ROW_A;        // 32 KB
constexpr int B_BYTES = HR * NCH * ROW_B;        // 8 KB
constexpr int SLOT_BYTES = A_BYTES + B_BYTES;
constexpr int NSTAGE = 5;
constexpr int SMEM_BYTES = NSTAGE * SLOT_BYTES + 1024;
static_assert(SMEM_BYTES <= 227 * 1024 && A_BYTES % 1024 == 0 && SLOT_BYTES % 1024 == 0, "ring");
}  // namespace gw16

template <typename T>
__global__ void __launch_bounds__(gw16::NT, 1)
sapa_gath_wide_16_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap, const Args a) {
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * gw16::NSTAGE];     // full, empty
    __shared__ int tile_ids[8];       // item of the ti-th turn at ti & 7, -1 = no more (the producer is at most NSTAGE turns ahead)
    const unsigned ring_addr = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned full_addr = (unsigned)__cvta_generic_to_shared(bars), empty_addr = full_addr + 8 * gw16::NSTAGE;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wy = warp & 3, wcol = warp >> 2, g = lane >> 2, t = lane & 3;
    const int sW = 2 * a.W;
    const size_t hi_plane = (size_t)(2 * a.H) * sW;
    const int nst = a.stages, nitems = a.B * a.tiles_x * a.tiles_y * a.csplit;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < gw16::NSTAGE; ++i) {
            mbar_init(full_addr + 8 * i, 1);
            mbar_init(empty_addr + 8 * i, gw16::NW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    begin_after_previous();

    if (warp >= gw16::NW) {           // producer: one lane; the stages of successive items form one stream through the ring
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;\n");
        if (tid != gw16::NW * 32) return;
        int slot = 0, phase = 0;
        for (int ti = 0;; ++ti) {
            int item = (int)blockIdx.x;
            if (ti > 0) item = (int)(atomicAdd(&g_next_tile[a.sched_slot], 1u) + gridDim.x);
            if (item >= nitems) item = -1;
            int x0 = 0, y0 = 0, n = 0, vb = 0;
            if (item >= 0) {
                int u = item;
                vb = u % a.csplit * nst; u /= a.csplit;
                x0 = (u % a.tiles_x) * gw16::COLS; u /= a.tiles_x;
                y0 = (u % a.tiles_y) * ROWS; n = u / a.tiles_y;
            }
            for (int it = 0; it < (item < 0 ? 1 : nst); ++it) {
                if (!mbar_wait_bounded(empty_addr + 8 * slot, phase ^ 1)) {
                    atomicExch(&g_wait_timeout, 1);
                    drain_loads<gw16::NSTAGE>(full_addr, slot, phase);
                    return;
                }
                const unsigned bar = full_addr + 8 * slot, dst = ring_addr + slot * gw16::SLOT_BYTES;
                if (it == 0) tile_ids[ti & 7] = item;
                if (item < 0) {
                    mbar_arrive(bar);          // completes the phase without data: the warps read -1 and stop
                } else {
                    mbar_expect_tx(bar, gw16::SLOT_BYTES);
                    tma_load_4d(dst, &amap, bar, 2 * x0 - 8, (vb + it) * gw16::NCH, 2 * (y0 - a.top - 2), n);
                    tma_load_4d(dst + gw16::A_BYTES, &bmap, bar, 2 * x0 + 56, (vb + it) * gw16::NCH, 2 * (y0 - a.top - 2), n);
                }
                if (++slot == gw16::NSTAGE) { slot = 0; phase ^= 1; }
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

    // ldmatrix rows of this lane: channel ch of the stage, high-res row r of a parent; chunk = 8 pixels = 16 bytes.  The warp reads the
    // chunks 2 wcol .. 2 wcol + 3 of the 80 pixels; chunks 8 and 9 are the second box.
    const int ch = (lane & 7) + 8 * ((lane >> 3) & 1), r = lane >> 4;
    int off[4], step[4];              // byte offset at parent row 0, bytes from one parent row to the next
#pragma unroll
    for (int kg = 0; kg < 4; ++kg) {
        const int chunk = 2 * wcol + kg;
        const bool second = chunk >= 8;
        step[kg] = 2 * gw16::NCH * (second ? gw16::ROW_B : gw16::ROW_A);
        off[kg] = second ? gw16::A_BYTES + (2 * wy + r) * gw16::NCH * gw16::ROW_B + ch * gw16::ROW_B + (((chunk - 8) ^ ((ch >> 2) & 1)) << 4)
                         : (2 * wy + r) * gw16::NCH * gw16::ROW_A + ch * gw16::ROW_A + ((chunk ^ (ch & 7)) << 4);
    }

    int slot = 0, phase = 0;
    for (int ti = 0;; ++ti) {
        if (!mbar_wait_bounded(full_addr + 8 * slot, phase)) { atomicExch(&g_wait_timeout, 1); return; }
        int item = tile_ids[ti & 7];              // published by the producer before the barrier's phase completed
        if (item < 0) break;
        int c0 = item % a.csplit * nst * gw16::NCH; item /= a.csplit;
        const int x0 = (item % a.tiles_x) * gw16::COLS + 8 * wcol; item /= a.tiles_x;     // first column of this warp
        const int y = (item % a.tiles_y) * ROWS + wy, n = item / a.tiles_y;
        // rows of length 8k: the warp's columns are inside the image together or not at all
        const bool live = y < a.Hout && x0 < a.W;
        // B fragments: W[px][col g] of the 5 parent rows x 4 chunks, [0] = upper, [1] = lower high-res row.  Parent row yp = y - 2 + j
        // uses window row 4 - j; the parent x0 - 4 + 4 kg + t of the pair reaches column x0 + g through window column g + 6 - 4 kg - t
        unsigned bw[5][4][2];
        const T *wimg = static_cast<const T *>(a.wt) + (size_t)n * 25 * hi_plane;
        // element of (j, kg): one step per parent row down is five planes back and two rows on, one per chunk four planes back
        const long long plane = (long long)hi_plane, w0 = (26 + g - t) * plane + 2 * (long long)(y - a.top - 2) * sW + 2 * x0 - 8 + 2 * t;
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const int yp = y - a.top - 2 + j;
            const bool row_in = live && yp >= 0 && yp < a.H;
#pragma unroll
            for (int kg = 0; kg < 4; ++kg) {
                const int dx = g + 6 - 4 * kg - t, hx = 2 * x0 - 8 + 8 * kg + 2 * t;
                const bool ok = row_in && dx >= 0 && dx <= 4 && hx >= 0 && hx < sW;
                const T *p = wimg + (ok ? w0 + j * (2 * (long long)sW - 5 * plane) + kg * (8 - 4 * plane) : 0);
                bw[j][kg][0] = ok ? *reinterpret_cast<const unsigned *>(p) : 0u;
                bw[j][kg][1] = ok ? *reinterpret_cast<const unsigned *>(p + sW) : 0u;
            }
        }
        const size_t out_plane = (size_t)a.Hout * a.W;
        T *o = static_cast<T *>(a.out) + ((size_t)n * a.C + c0 + g) * out_plane + (size_t)y * a.W + x0 + 2 * t;
        for (int it = 0; it < nst; ++it, c0 += gw16::NCH, o += (size_t)gw16::NCH * out_plane) {
            if (it > 0 && !mbar_wait_bounded(full_addr + 8 * slot, phase)) { atomicExch(&g_wait_timeout, 1); return; }
            const unsigned stage = ring_addr + slot * gw16::SLOT_BYTES;
            float acc[4][4] = {};                 // one chain per chunk
            if (live) {
#pragma unroll
                for (int j = 0; j < 5; ++j)
#pragma unroll
                    for (int kg = 0; kg < 4; ++kg) {
                        unsigned x[4];
                        ldsm_x4(x, stage + off[kg] + j * step[kg]);
                        mma_h16<T>(acc[kg], x[0], x[1], x[2], x[3], bw[j][kg][0], bw[j][kg][1]);
                    }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty_addr + 8 * slot);
            if (++slot == gw16::NSTAGE) { slot = 0; phase ^= 1; }
            if (live) {                           // D fragment: d0, d1 = G[ch g][cols 2t, 2t + 1], d2, d3 = G[ch g + 8][same]
                float s[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i] = (acc[0][i] + acc[1][i]) + (acc[2][i] + acc[3][i]);
                if (c0 + g < a.C) *reinterpret_cast<unsigned *>(o) = pack_pair(T(), s[0], s[1]);
                if (c0 + 8 + g < a.C) *reinterpret_cast<unsigned *>(o + 8 * out_plane) = pack_pair(T(), s[2], s[3]);
                if (!((s[0] + s[1] + s[2] + s[3]) * 0.f == 0.f)) store_cell_sums<T>(a, n, c0 + g, 2, y, x0 + 2 * t);
            }
        }
    }
}
