// sapa_strip_fwd.cuh — the fused forward in 16 bits (K = 5, s = 2, up to 64 query channels) on strips of 32 low-res columns, both products
// on the 5th-generation tensor cores.  Included by sapa_tma.cu behind sapa_strip.cuh, whose aggregation this is; here the weights are
// computed:
//   * logits: for one low-res row, its 128 high-res pixels are the lanes of ONE product
//         S[128 px x 48 cells] = Q^T[128 px x d] * K[d x 48 cells]
//     per window row; query and key boxes are the operands as TMA lands them (channel rows of 128 bytes: "MN-major", 128-byte swizzle).  A
//     row of keys stays in shared memory for the five steps that use it.  Window rows 0 to 2 and 3, 4 are handed over by themselves: the
//     next step's logits of a part are computed as soon as this step's have been read (handed over as a whole, that chain was what the
//     kernel waited for).
//   * softmax: a thread holds a pixel: it reads the 20 cells that its warp's pixels reach, shifts its own five to the front (their place
//     depends on the lane) and has the 25 logits of its pixel in registers; no shuffles, no shared memory.  The weights go to the
//     banded operand P of the aggregation, and to the attention map where it is asked for.  Two warpgroups take turns.
//   * the aggregation's accumulator is two halves (16 parents each), drained by a warpgroup each while the other half is computed.
// The logits of a step are computed while the step before is aggregated; a warp each issues the two kinds of MMAs (one for both could not
// issue them fast enough: 64 x 32 x 32x32 27.8 us, 18.4 with two).  Blocks of 128 value channels compute their logits anew.
// Values that are not finite stay out of the product (finite.cuh) and reach the pixels whose windows hold them; an infinity comes to what its 16-bit weight
// makes of it.
// What bounds it: loads in flight, and memory (64 x 256 x 128x128, bfloat16: 700 us, 4.8 TB/s; 824 on tiles, whose ldmatrix wavefronts and MMA
// issue bound them).  Prefetches of the next rows into L2 make it slower (830).
namespace sfwd {

using namespace ummau;
using strip::CH; using strip::VROW; using strip::VCHUNKS; using strip::ACOLS; using strip::Item; using strip::SArgs;

constexpr int EPI_WARPS = 8, SPLIT_WARP0 = 8, SOFT_WARP0 = 12, QK_WARP = 20, S_WARP = 21, MMA_WARP = 22, V_WARP = 23, NT = 24 * 32;
constexpr int V_BYTES = CH * VROW, MAX_NVL = 4;             // landed rows of V
constexpr int MAX_D = 64, MAX_NKR = 10, MAX_NQ = 4;         // query channels; rows of keys, steps of queries in shared memory
constexpr int CELLS = 32, SN = 48;                          // low-res columns of a strip; cells of a row of logits (columns x0 - 8 and so on)
constexpr int NV = 6, NP = 2;
constexpr int S_COL = 0, D_COL = 5 * SN, V_COL = D_COL + 4 * CELLS, TMEM_COLS = 512;
constexpr int OUT_BYTES = 2 * 32 * 128;                     // of a pair of epilogue warps: [high-res row][channel][pixel]
static_assert(V_COL + NV * ACOLS <= TMEM_COLS, "tensor memory");
template <typename T, int KSTEPS> struct Lay {
    using G = strip::Geo<T>;
    // five rows of keys and one step of queries are in use, the others on their way, as shared memory allows: 64 x 256 x 128x128, 64 query channels:
    // 6 rows, 2 steps and 3 rows of values 739 us, 7, 2 and 3 737, 7, 3 and 2 687 to 700
    static constexpr int KROW = KSTEPS * 16 * 128, NKR = KSTEPS == 4 ? 7 : KSTEPS == 3 ? 8 : 10, NQ = KSTEPS == 4 ? 3 : 4, NVL = KSTEPS == 4 ? 2 : KSTEPS == 3 ? 3 : 4;
    static constexpr int OUT0 = 0, K0 = 4 * OUT_BYTES, Q0 = K0 + NKR * KROW, V0 = Q0 + NQ * 2 * KROW, P0 = V0 + NVL * V_BYTES;
    static constexpr int SMEM = P0 + NP * G::P_BYTES + 1024;
    static_assert(SMEM <= 227 * 1024 && G::CELLS == CELLS, "layout");
};
struct FArgs {
    SArgs s;
    void *attn;            // optional output
    const void *q, *k;     // for outputs with an infinity in their windows
    int d;
};
__device__ __forceinline__ void tc_ld4(unsigned taddr, unsigned *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
// Window slots whose 16-bit weight for a pixel is zero (or NaN), formed again by a warp, a slot to a lane
template <typename T> __device__ __forceinline__ unsigned no_weight(const FArgs &f, int n, int hy, int hx, int lane) {
    const SArgs &a = f.s;
    const size_t hi_plane = (size_t)(2 * a.H) * (2 * a.W), lo_plane = (size_t)a.rows * a.W;
    const int y = a.ytop0 + (hy >> 1) + lane / 5 - 2, x = (hx >> 1) + lane % 5 - 2;
    const bool slot = lane < 25, cell = slot && y >= 0 && y < a.rows && x >= 0 && x < a.W;
    const T *q = static_cast<const T *>(f.q) + (size_t)n * f.d * hi_plane + (size_t)hy * (2 * a.W) + hx;
    const T *k = static_cast<const T *>(f.k) + (size_t)n * f.d * lo_plane + (cell ? (size_t)y * a.W + x : 0);
    float s = 0.f;
#pragma unroll 4
    for (int c = 0; c < f.d; ++c) s = fmaf(to_acc(q[c * hi_plane]), cell ? to_acc(k[c * lo_plane]) : 0.f, s);
    float m = slot ? s : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float e = slot ? expf(s - m) : 0.f;
    float z = e;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
    return __ballot_sync(0xffffffffu, slot && !(to_acc(from_acc<T>(e / z)) > 0.f));
}
// Outputs of half a strip's row with something not finite in their windows, which the products took as zero, once they are stored: NaN next to a NaN,
// to infinities of both signs and to one whose weight is zero.  By a whole warp.  dy0, dy1: the window rows that may hold such elements.
template <typename T> __device__ __noinline__ void finish_pixels(const FArgs &f, int n, int x0, int c, int y, int half, int dy0, int dy1, int lane) {
    const SArgs &a = f.s;
    constexpr int FIRST = strip::Geo<T>::BOX0 - 2;                    // bit of a parent's first column
    const unsigned mine = 0xffffu << (16 * half);
    unsigned nan = 0u;                                                // parents next to a NaN
    unsigned long long up[5], down[5];
#pragma unroll
    for (int dy = 0; dy < 5; ++dy) {
        finite::Marks m{0ull, 0ull, 0ull};
        if (c < a.C && dy >= dy0 && dy <= dy1 && (nan & mine) != mine) m = strip::marks_of<T>(a, n, c, y, dy, x0);
        nan |= (unsigned)strip::reached<T>(m.nan); up[dy] = m.up; down[dy] = m.down;
    }
    const size_t hi_plane = (size_t)(2 * a.H) * (2 * a.W);
    T *const out = static_cast<T *>(a.out) + ((size_t)n * a.C + c) * hi_plane + (size_t)(2 * y) * (2 * a.W) + 2 * x0;
#pragma unroll 1
    for (int p = 16 * half; p < 16 * half + 16 && x0 + p < a.W; ++p) {
        if ((p & 3) == 0 && __all_sync(0xffffffffu, c >= a.C || (nan >> p & 15) == 15)) {      // 16 bytes of each row
            if (c < a.C) *reinterpret_cast<uint4 *>(out + 2 * p) = *reinterpret_cast<uint4 *>(out + 2 * a.W + 2 * p) = finite::nan_chunk<T>();
            p += 3;
            continue;
        }
        unsigned ups = 0u, downs = 0u;                                // window slots
#pragma unroll
        for (int dy = 0; dy < 5; ++dy) {
            ups |= (unsigned)(up[dy] >> (FIRST + p) & 31) << (5 * dy);
            downs |= (unsigned)(down[dy] >> (FIRST + p) & 31) << (5 * dy);
        }
        const bool none = (nan >> p & 1) != 0u || (ups != 0u && downs != 0u), some = (ups | downs) != 0u;
        if (!__any_sync(0xffffffffu, none || some)) continue;
        const bool ask = __any_sync(0xffffffffu, some && !none);
#pragma unroll 1
        for (int e = 0; e < 4; ++e) {
            const int r = e >> 1, px = 2 * p + (e & 1);
            const unsigned gone = ask ? no_weight<T>(f, n, 2 * y + r, 2 * x0 + px, lane) : 0u;
            if (!none && !some) continue;
            const float s = none || ((ups | downs) & gone) != 0u ? finite::nan_value() : ups != 0u ? INFINITY : -INFINITY;
            out[(size_t)r * (2 * a.W) + px] = from_acc<T>(s);
        }
    }
}
// the steps (rows) of a CTA's items, one after the other
template <typename T> struct Cursor {
    Item t;
    int i, y;
    bool more;
    __device__ __forceinline__ Cursor(const SArgs &a, int items) : i((int)blockIdx.x), more(i < items) {
        if (more) { t = strip::item_at<T>(a, i); y = t.y0; }
    }
    __device__ __forceinline__ void next(const SArgs &a, int items) {
        if (++y < t.y1) return;
        i += gridDim.x;
        more = i < items;
        if (more) { t = strip::item_at<T>(a, i); y = t.y0; }
    }
};
}  // namespace sfwd

template <typename T, int KSTEPS>
__global__ void __launch_bounds__(sfwd::NT, 1) sapa_strip_fwd_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                                                                     const __grid_constant__ CUtensorMap vmap, const __grid_constant__ CUtensorMap omap,
                                                                     const __grid_constant__ sfwd::FArgs f) {
    using namespace sfwd;
    using G = strip::Geo<T>;
    using L = Lay<T, KSTEPS>;
    constexpr int NKR = L::NKR, NQ = L::NQ, NVL = L::NVL;
    const SArgs &a = f.s;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * (sfwd::MAX_NVL + sfwd::NV + MAX_NKR + MAX_NQ + sfwd::NP + 2) + 6];
    __shared__ unsigned tmem_slot;
    __shared__ finite::Noted noted;                                   // rows of V, counted over the CTA's items
    const unsigned base = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned vfull = (unsigned)__cvta_generic_to_shared(bars), vempty = vfull + 8 * NVL, aready = vempty + 8 * NVL, aempty = aready + 8 * sfwd::NV;
    const unsigned kfull = aempty + 8 * sfwd::NV, kempty = kfull + 8 * NKR, qfull = kempty + 8 * NKR, qempty = qfull + 8 * NQ;
    const unsigned pready = qempty + 8 * NQ, pempty = pready + 8 * sfwd::NP, dfull = pempty + 8 * sfwd::NP, dempty = dfull + 16, sfull = dempty + 16, sempty = sfull + 32;
    const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
    const int items = a.B * a.cblocks * a.segs * a.strips;

    if (tid < 4) noted.clear(tid);
    if (tid == 0) {
        for (int i = 0; i < NVL; ++i) { mbar_init(vfull + 8 * i, 1); mbar_init(vempty + 8 * i, 128); }
        for (int i = 0; i < sfwd::NV; ++i) { mbar_init(aready + 8 * i, 128); mbar_init(aempty + 8 * i, 1); }
        for (int i = 0; i < NKR; ++i) { mbar_init(kfull + 8 * i, 1); mbar_init(kempty + 8 * i, 1); }
        for (int i = 0; i < NQ; ++i) { mbar_init(qfull + 8 * i, 1); mbar_init(qempty + 8 * i, 1); }
        for (int i = 0; i < sfwd::NP; ++i) { mbar_init(pready + 8 * i, 128); mbar_init(pempty + 8 * i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(dfull + 8 * i, 1); mbar_init(dempty + 8 * i, 128); }
        for (int i = 0; i < 4; ++i) mbar_init(sfull + 8 * i, 1);      // [warpgroup that takes the step][part]
        for (int i = 0; i < 2; ++i) mbar_init(sempty + 8 * i, 128);   // of a part
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == sfwd::MMA_WARP) {
        tc_alloc((unsigned)__cvta_generic_to_shared(&tmem_slot), sfwd::TMEM_COLS);
        tc_relinquish();
    }
    for (int i = tid; i < sfwd::NP * G::P_BYTES / 16; i += sfwd::NT)
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(base + L::P0 + 16 * i), "r"(0u) : "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = warp_uniform(*reinterpret_cast<volatile unsigned *>(&tmem_slot));
    const unsigned quarter = (unsigned)((warp & 3) * 32) << 16;       // the lanes of tensor memory that a warp can reach
    unsigned zeros[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) zeros[i] = 0u;
    if (warp < sfwd::EPI_WARPS) {
#pragma unroll 1
        for (int c = 0; c < 64; c += 16) tc_st16(tmem + quarter + D_COL + (warp >> 2) * 64 + c, zeros);
        tc_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    begin_after_previous();

    bool ok = true;
    if (warp == QK_WARP) {
        if (lane == 0) {
            int ks = 0, kph = 0, qs = 0, qph = 0;
            constexpr int row_bytes = L::KROW;
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item t = strip::item_at<T>(a, i);
                for (int y = t.y0 - 2; y < t.y1 + 2 && ok; ++y) {
                    if (!mbar_wait_bounded(kempty + 8 * ks, kph ^ 1)) { ok = false; break; }
                    mbar_expect_tx(kfull + 8 * ks, row_bytes);
                    tma_load_4d(base + L::K0 + ks * L::KROW, &kmap, kfull + 8 * ks, t.x0 - 8, 0, a.ytop0 + y, t.n);
                    if (++ks == NKR) { ks = 0; kph ^= 1; }
                    if (y < t.y0 + 2) continue;
                    if (!mbar_wait_bounded(qempty + 8 * qs, qph ^ 1)) { ok = false; break; }
                    mbar_expect_tx(qfull + 8 * qs, 2 * row_bytes);
                    tma_load_4d(base + L::Q0 + qs * 2 * L::KROW, &qmap, qfull + 8 * qs, 2 * t.x0, 0, 2 * (y - 2), t.n);
                    if (++qs == NQ) { qs = 0; qph ^= 1; }
                }
            }
            if (!ok) {                                                // none of its loads may land after it has left
                (void)drain_loads<NKR>(kfull, ks, kph);
                (void)drain_loads<NQ>(qfull, qs, qph);
            }
        }
    } else if (warp == V_WARP) {
        if (lane == 0) {
            int vs = 0, vph = 0;
            const int vbytes = min(a.C, CH) * VROW;
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item t = strip::item_at<T>(a, i);
                for (int y = t.y0 - 2; y < t.y1 + 2; ++y) {
                    if (!mbar_wait_bounded(vempty + 8 * vs, vph ^ 1)) { ok = false; break; }
                    mbar_expect_tx(vfull + 8 * vs, vbytes);
                    tma_load_4d(base + L::V0 + vs * sfwd::V_BYTES, &vmap, vfull + 8 * vs, t.x0 - G::BOX0, t.c0, a.ytop0 + y, t.n);
                    if (++vs == NVL) { vs = 0; vph ^= 1; }
                }
            }
            if (!ok) (void)drain_loads<NVL>(vfull, vs, vph);
        }
    } else if (warp == S_WARP) {
        constexpr unsigned HI_QK = (1024u >> 4) | (1u << 14) | (2u << 29);      // keys, queries: 8 channels of 128 bytes, 128-byte swizzle
        constexpr unsigned IDESC_S = IDESC_M128<T> | (1u << 15) | (1u << 16) | idesc_n(SN);        // both operands MN-major
        constexpr unsigned ROW = L::KROW >> 4;            // a row of keys, half a step of queries
        const unsigned leader = elect_leader();
        const unsigned k_base = warp_uniform(desc_lo(base + L::K0, L::KROW)), k_end = k_base + NKR * ROW, q_base = warp_uniform(desc_lo(base + L::Q0, L::KROW));
        // ring positions advance by one with a wrap: a remainder per product would be computed outside the uniform registers
        int k0 = 0, kin = 0, kslot = 0, kph = 0, qs = 0, qph = 0, step = 0;        // slot of window row 0; rows waited for
        Cursor<T> c(a, items);
        while (c.more && ok) {
            for (; kin < 5 && ok; ++kin) {
                ok = mbar_wait_warp(kfull + 8 * kslot, kph);
                if (++kslot == NKR) { kslot = 0; kph ^= 1; }
            }
            ok = ok && mbar_wait_warp(qfull + 8 * qs, qph);
            unsigned k = k_base + k0 * ROW;
            const unsigned q = q_base + qs * (2 * ROW);
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {
                if (dy == 0 || dy == 3) {                             // the part of the step before has been read
                    ok = ok && mbar_wait_warp(sempty + dy / 3 * 8, (step & 1) ^ 1);
                    if (!ok) break;
                    tc_fence_after();
                }
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks)
                    tc_mma<false>(leader, tmem + S_COL + dy * SN, q + ks * (2048 >> 4), k + ks * (2048 >> 4), HI_QK, IDESC_S, ks > 0 ? 1u : 0u);
                k += ROW;
                if (k == k_end) k = k_base;
                if (dy == 2 || dy == 4) tc_commit_by(leader, sfull + 16 * (step & 1) + dy / 3 * 8);
            }
            if (!ok) break;
            ++step;
            tc_commit_by(leader, qempty + 8 * qs);
            if (++qs == NQ) { qs = 0; qph ^= 1; }
            for (int e = c.y == c.t.y1 - 1 ? 5 : 1; e > 0; --e) {     // the row that no later step uses; of an item's last step all five
                tc_commit_by(leader, kempty + 8 * k0);
                --kin;
                if (++k0 == NKR) k0 = 0;
            }
            c.next(a, items);
        }
    } else if (warp == sfwd::MMA_WARP) {
        constexpr unsigned HI = (128u >> 4) | (1u << 14);             // P: 8-row groups 128 bytes apart, descriptor version 1, no swizzle
        const unsigned leader = elect_leader(), p_base = warp_uniform(base + L::P0);
        const unsigned b0 = desc_lo(p_base + G::tile(0), G::lbo(0)), b1 = desc_lo(p_base + G::tile(1), G::lbo(1)), b2 = desc_lo(p_base + G::tile(2), G::lbo(2));
        int v0 = 0, vin = 0, vslot = 0, vph = 0, dph = 0, pb = 0, pph = 0;
        Cursor<T> now(a, items);
        while (now.more && ok) {
            for (; vin < 5 && ok; ++vin) {
                ok = mbar_wait_warp(aready + 8 * vslot, vph);
                if (++vslot == sfwd::NV) { vslot = 0; vph ^= 1; }
            }
            ok = ok && mbar_wait_warp(pready + 8 * pb, pph);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                ok = ok && mbar_wait_warp(dempty + 8 * h, dph ^ 1);
                if (!ok) break;
                tc_fence_after();
                const unsigned pofs = (unsigned)(pb * G::P_BYTES) >> 4, d = tmem + D_COL + 64 * h, v_end = tmem + V_COL + sfwd::NV * ACOLS;
                unsigned ka = tmem + V_COL + v0 * ACOLS;
#pragma unroll
                for (int dy = 0; dy < 5; ++dy) {
                    const unsigned kb = pofs + ((dy * G::DY_BYTES) >> 4);
                    if (h == 0) {                                     // parents 0 .. 15
                        tc_mma_ta<false>(leader, d, ka, b0 + kb, HI, IDESC_M128<T> | idesc_n(64), 1u);
                        tc_mma_ta<false>(leader, d + 4 * G::p0(1), ka + 8, b1 + kb, HI, IDESC_M128<T> | idesc_n(4 * (16 - G::p0(1))), 1u);
                    } else {
                        tc_mma_ta<false>(leader, d, ka + 8, b1 + kb + 4 * (16 - G::p0(1)), HI, IDESC_M128<T> | idesc_n(64), 1u);
                        tc_mma_ta<false>(leader, d + 4 * (G::p0(2) - 16), ka + 16, b2 + kb, HI, IDESC_M128<T> | idesc_n(G::rows(2)), 1u);
                    }
                    ka += ACOLS;
                    if (ka == v_end) ka = tmem + V_COL;
                }
                tc_commit_by(leader, dfull + 8 * h);
            }
            if (!ok) break;
            dph ^= 1;
            tc_commit_by(leader, pempty + 8 * pb);
            if (++pb == sfwd::NP) { pb = 0; pph ^= 1; }
            for (int e = now.y == now.t.y1 - 1 ? 5 : 1; e > 0; --e) {
                tc_commit_by(leader, aempty + 8 * v0);
                --vin;
                if (++v0 == sfwd::NV) v0 = 0;
            }
            now.next(a, items);
        }
    } else if (warp >= SPLIT_WARP0 && warp < SOFT_WARP0) {
        int vs = 0, vph = 0, as = 0, aph = 0, row = 0;
        const unsigned line = ((warp & 3) * 32 + lane) * VROW;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = strip::item_at<T>(a, i);
            const bool used = t.c0 + (warp & 3) * 32 < a.C;           // lanes without a channel keep whatever they hold
            for (int y = t.y0 - 2; y < t.y1 + 2; ++y, ++row) {
                if (!mbar_wait_warp(vfull + 8 * vs, vph)) { ok = false; break; }
                unsigned v[4 * VCHUNKS];
                if (used) {
#pragma unroll
                    for (int q = 0; q < G::LOADS; ++q)
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[4 * q]), "=r"(v[4 * q + 1]), "=r"(v[4 * q + 2]), "=r"(v[4 * q + 3])
                                     : "r"(base + L::V0 + vs * sfwd::V_BYTES + line + 16 * q) : "memory");
                }
                if (!mbar_wait_warp(aempty + 8 * as, aph ^ 1)) { ok = false; break; }
                tc_fence_after();
                if (used) strip::move_cells<T>(tmem + quarter + V_COL + as * ACOLS, v, t.c0 + (warp & 3) * 32 + lane < a.C, noted, warp & 3, row, vempty + 8 * vs);
                else mbar_arrive(vempty + 8 * vs);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(aready + 8 * as);
                if (++vs == NVL) { vs = 0; vph ^= 1; }
                if (++as == sfwd::NV) { as = 0; aph ^= 1; }
            }
        }
    } else if (warp >= SOFT_WARP0 && warp < QK_WARP) {
        // thread = lane of S: pixel px of high-res row r
        const int group = (warp - SOFT_WARP0) >> 2, r = (warp >> 1) & 1, px = (warp & 1) * 32 + lane, parent = px >> 1, shift = lane >> 1;
        const bool odd = parent & 1;
        const int n = 4 * parent + 2 * r + (px & 1);
        unsigned to[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) to[e] = base + L::P0 + group * G::P_BYTES + G::at(n, (parent & ~1) + 2 * e);
        const unsigned from = tmem + quarter + S_COL + (warp & 1) * 16 + 6;
        const size_t hi_plane = (size_t)(2 * a.H) * (2 * a.W);
        constexpr float LOG2E = 1.4426950408889634f;
        int step = 0, ph = 0;
        Cursor<T> c(a, items);
        for (; c.more && ok; c.next(a, items), ++step) {
            if ((step & 1) != group) continue;
            float s[25];
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {
                if (dy == 3) { tc_fence_before(); mbar_arrive(sempty); }                  // the first part has been read
                if (dy == 0 || dy == 3) {
                    if (!mbar_wait_warp(sfull + 16 * group + 8 * (dy / 3), ph)) { ok = false; break; }
                    tc_fence_after();
                }
                unsigned w[20];
                tc_ld16(from + dy * SN, *reinterpret_cast<unsigned (*)[16]>(&w[0]));
                tc_ld4(from + dy * SN + 16, &w[16]);
                tc_wait_ld();
#pragma unroll
                for (int e = 0; e < 12; ++e) w[e] = shift & 8 ? w[e + 8] : w[e];
#pragma unroll
                for (int e = 0; e < 8; ++e) w[e] = shift & 4 ? w[e + 4] : w[e];
#pragma unroll
                for (int e = 0; e < 6; ++e) w[e] = shift & 2 ? w[e + 2] : w[e];
#pragma unroll
                for (int e = 0; e < 5; ++e) s[5 * dy + e] = __uint_as_float(shift & 1 ? w[e + 1] : w[e]);
            }
            if (!ok) break;
            tc_fence_before();
            mbar_arrive(sempty + 8);
            // exp(x - m) = 2^(x * log2(e) - m * log2(e)): one FMA and one ex2 per element
            float m = s[0], z = 0.f;
#pragma unroll
            for (int k = 1; k < 25; ++k) m = fmaxf(m, s[k]);
            m *= LOG2E;
#pragma unroll
            for (int k = 0; k < 25; ++k) s[k] = ex2_ftz(fmaf(s[k], LOG2E, -m));
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) z += ((s[5 * dy] + s[5 * dy + 1]) + (s[5 * dy + 2] + s[5 * dy + 3])) + s[5 * dy + 4];
            const float inv = __frcp_rn(z);
#pragma unroll
            for (int k = 0; k < 25; ++k) s[k] *= inv;
            if (!mbar_wait_warp(pempty + 8 * group, ph ^ 1)) { ok = false; break; }
            ph ^= 1;
#pragma unroll
            for (int dy = 0; dy < 5; ++dy) {                          // cell pairs start at even cells
                const float *w = s + 5 * dy;
                sts32(to[0] + dy * G::DY_BYTES, odd ? pack_pair(T(), 0.f, w[0]) : pack_pair(T(), w[0], w[1]));
                sts32(to[1] + dy * G::DY_BYTES, odd ? pack_pair(T(), w[1], w[2]) : pack_pair(T(), w[2], w[3]));
                sts32(to[2] + dy * G::DY_BYTES, odd ? pack_pair(T(), w[3], w[4]) : pack_pair(T(), w[4], 0.f));
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            mbar_arrive(pready + 8 * group);
            if (f.attn != nullptr && c.t.c0 == 0 && c.t.x0 + parent < a.W) {
                T *an = static_cast<T *>(f.attn) + (size_t)c.t.n * 25 * hi_plane + (size_t)(2 * c.y + r) * (2 * a.W) + 2 * c.t.x0 + px;
#pragma unroll
                for (int k = 0; k < 25; ++k) an[k * hi_plane] = from_acc<T>(s[k]);
            }
        }
    } else if (warp < sfwd::EPI_WARPS) {
        // warps w and w + 4 share an output box: the halves of the strip's columns
        const int half = warp >> 2;
        const unsigned box = base + L::OUT0 + (warp & 3) * sfwd::OUT_BYTES, stage = box + lane * 128, d = tmem + quarter + D_COL + 64 * half;
        int dph = 0;
        auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (warp & 3)) : "memory"); };
        Cursor<T> c(a, items);
        for (; c.more; c.next(a, items)) {
            const int cw = c.t.c0 + (warp & 3) * 32;
            ok = ok && mbar_wait_warp(dfull + 8 * half, dph);         // a warp that gives up goes on to its partner's barriers
            dph ^= 1;
            tc_fence_after();
            if (half == 0 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");       // the last store has read the box
            __syncwarp();
            pair_sync();
#pragma unroll
            for (int g = 0; g < 2; ++g) {                             // 8 parents at a time: 16 pixels of both high-res rows
                unsigned v[32];
                tc_ld16(d + 32 * g, *reinterpret_cast<unsigned (*)[16]>(&v[0]));
                tc_ld16(d + 32 * g + 16, *reinterpret_cast<unsigned (*)[16]>(&v[16]));
                tc_wait_ld();
                tc_st16(d + 32 * g, zeros);
                tc_st16(d + 32 * g + 16, zeros);
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        auto px = [&](int e) { return __uint_as_float(v[4 * ((q * 8 + e) >> 1) + 2 * r + (e & 1)]); };
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(stage + r * (32 * 128) + (((4 * half + 2 * g + q) ^ (lane & 7)) << 4)),
                                     "r"(pack_pair(T(), px(0), px(1))), "r"(pack_pair(T(), px(2), px(3))), "r"(pack_pair(T(), px(4), px(5))),
                                     "r"(pack_pair(T(), px(6), px(7))) : "memory");
                    }
            }
            tc_wait_st();
            tc_fence_before();
            if (ok) mbar_arrive(dempty + 8 * half);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            pair_sync();
            if (half == 0 && lane == 0 && cw < a.C && ok) {           // pixels and channels beyond the tensor are cut off
                tma_store_4d(&omap, box, 2 * c.t.x0, cw, 2 * c.y, c.t.n);
                tma_store_4d(&omap, box + 32 * 128, 2 * c.t.x0, cw, 2 * c.y + 1, c.t.n);
                asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
    if (!ok) atomicExch(&g_wait_timeout, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == sfwd::MMA_WARP) tc_dealloc(tmem, sfwd::TMEM_COLS);
    if (warp < sfwd::EPI_WARPS && noted.last[warp & 3] >= 0) {        // rare: outputs with something not finite (all are stored)
        const int first = noted.first[warp & 3], last = noted.last[warp & 3];
        int row = 0;
        for (Cursor<T> c(a, items); c.more; c.next(a, items)) {
            if (row + 4 >= first && row <= last)
                finish_pixels<T>(f, c.t.n, c.t.x0, c.t.c0 + (warp & 3) * 32 + lane, c.y, warp >> 2, first - row, last - row, lane);
            row += c.y == c.t.y1 - 1 ? 5 : 1;
        }
    }
}
