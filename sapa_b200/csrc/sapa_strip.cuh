// sapa_strip.cuh — the aggregation out[c][p] = sum over window slots k of  Wt[k][p] * V[c][win_k(p)]  (K = 5, s = 2) on the 5th-generation
// tensor cores.  Included by sapa_tma.cu, inside namespace sapa::tma.
//
// A CTA walks a strip of low-res columns (16 in float32, 32 in 16 bits) down the image for 128 channels, one low-res row = two high-res
// rows at a time:
//     D[128 ch x (4 x strip) px] = sum over the five window rows of  V[128 ch x K cells] * P[K cells x (4 x strip) px]
//   * V: one TMA box (128 channels x 112 bytes of one row: an odd number of 16-byte chunks, read without bank conflicts) per row.  A
//     warpgroup moves it into a ring of rows in tensor memory as the A operand (lane = channel, column = 32 bits of cells), where five
//     products use it; float32 is split on the way into the terms of the three-term tf32 product.
//   * P: the banded operand of a step, 15 tiles (window row, 32 bytes of cells) of the pixels that the cells reach: a third of the band is
//     not zero.  Its zeros are the same in every step and are written once; two warpgroups overwrite the 25 weights per pixel.
//     Pixels are ordered parent by parent, so that the pixels of a tile are consecutive columns of D.
//   * one warp issues the MMAs (N = 16 to 80, N / 2 clocks each), in float32, with three times as many, one for each half of the strip: a warp issues
//     an MMA in about 26 clocks (32 x 64 x 64x64 58 us with one, 54 with two).  float32 adds the small products first, because an accumulation in
//     tensor memory rounds toward zero: eight roundings of the whole sum instead of twenty-four.
//   * epilogue: tcgen05.ld (lane = channel), zeros back into D, rows of 128 bytes through shared memory, TMA stores; a warpgroup for each of
//     the two accumulators (with one for both it was what the kernel waited for: 32 x 64 x 64x64, bfloat16, 45 -> 32 us).
//   * what is not finite stays out of the products (finite.cuh); a second pass over the rows in question forms the outputs that it reaches.  Formed in
//     the epilogue, output by output, they took one NaN in the values from 19 to 640 us and a tensor of NaN to 6.8 ms; now 58 and 125 (8 x 256 x
//     64x64, bfloat16).
// The kernels on tiles load (and split) a value fragment once per window row and group of pixels that it reaches; their fragment loads, splits
// and mma.sync issue bound them.  What bounds this one: memory (8 x 256 x 64x64: float32 54 -> 37 us, 4.9 TB/s of reads and mostly writes;
// bfloat16 30 -> 18, 5.1 TB/s), with few channels the MMAs and the epilogue, which work on 128 lanes (32 x 64 x 64x64: 76 -> 51, 42 -> 26).
namespace strip {

using namespace ummau;

constexpr int CH = 128;                                     // channels of an item = lanes of tensor memory
constexpr int EPI_WARPS = 8, SPLIT_WARP0 = 8, P_WARP0 = 12, P_WARPS = 8, TMA_WARP = 20, MMA_WARP = 21, NT = 23 * 32;
constexpr int VROW = 112, VCHUNKS = 7, ACOLS = 24;          // bytes and 16-byte chunks of a box row; columns of an A operand (one term)
constexpr int V_BYTES = CH * VROW, NVL = 4;                 // landed rows of V
constexpr int L_BYTES = 2 * 25 * 128, NWL = 4;              // landed weights: [high-res row][slot][pixel]
constexpr int NV = 8, ND = 2, NP = 2;                       // rows of V in tensor memory, accumulators, operands P
constexpr int OUT_BYTES = 2 * 32 * 128;                     // of an epilogue warp: [high-res row][channel][pixel]
constexpr int TMEM_COLS = 512;

template <typename T> struct Geo {
    static constexpr bool F32 = sizeof(T) == 4;
    static constexpr int CELLS = F32 ? 16 : 32, PX = 2 * CELLS, N = 4 * CELLS;
    static constexpr int KS = 32 / (int)sizeof(T);          // cells of an MMA
    static constexpr int TERMS = F32 ? 2 : 1;
    static constexpr int SHIFT = F32 ? 2 : 3;               // words from the box's start (16-byte boundary) to cell x0 - 2, the first of the product
    static constexpr int BOX0 = F32 ? 4 : 8;                // the box starts at column x0 - BOX0
    static constexpr int ABUF = TERMS * ACOLS;
    // words of a row that windows reach (float32: all, zeros for the last four cost 32 x 64 x 64x64 51.7 -> 53.0 us), and the landed chunks that hold them
    static constexpr int WORDS = F32 ? ACOLS : (CELLS + 4) * (int)sizeof(T) / 4;
    static constexpr int LOADS = (SHIFT + WORDS + 3) / 4;
    static constexpr int ISSUERS = F32 ? 2 : 1;             // warps that issue the MMAs, each those of half of the strip's parents
    // K step j: parents [p0, p1) of the strip reach its cells (columns x0 - 2 + KS j and so on)
    __host__ __device__ static constexpr int p0(int j) { return KS * j < 4 ? 0 : KS * j - 4; }
    __host__ __device__ static constexpr int p1(int j) { return KS * j + KS < CELLS ? KS * j + KS : CELLS; }
    __host__ __device__ static constexpr int rows(int j) { return 4 * (p1(j) - p0(j)); }
    __host__ __device__ static constexpr int lbo(int j) { return rows(j) * 16 + 64; }       // + 64: the two chunks of a tile start in different banks
    __host__ __device__ static constexpr int tile(int j) { return j == 0 ? 0 : j == 1 ? 2 * lbo(0) : 2 * lbo(0) + 2 * lbo(1); }
    static constexpr int DY_BYTES = 2 * (lbo(0) + lbo(1) + lbo(2)), P_TERM = 5 * DY_BYTES, P_BYTES = TERMS * P_TERM;
    static constexpr int OUT0 = 0, V0 = EPI_WARPS * OUT_BYTES, L0 = V0 + NVL * V_BYTES, P0 = L0 + NWL * L_BYTES;
    static constexpr int SMEM = P0 + NP * P_BYTES + 1024;
    static_assert(ND * N + NV * ABUF <= TMEM_COLS && SMEM <= 227 * 1024 && p1(2) == CELLS && rows(0) % 16 == 0 && rows(1) % 16 == 0 && rows(2) % 16 == 0, "layout");
    // byte offset of (pixel column n, cell) in a term of P for window row 0; cell = parent + dx of the strip
    static __device__ __forceinline__ int at(int n, int cell) {
        const int j = cell / KS, in = cell % KS;
        const int p = j == 0 ? p0(0) : j == 1 ? p0(1) : p0(2), l = j == 0 ? lbo(0) : j == 1 ? lbo(1) : lbo(2), base = j == 0 ? tile(0) : j == 1 ? tile(1) : tile(2);
        return base + in / (KS / 2) * l + (n - 4 * p) * 16 + in % (KS / 2) * (int)sizeof(T);
    }
};

struct SArgs {
    const void *v, *wt;    // for outputs with something not finite in their windows
    void *out;
    int B, C, H, W, rows, ytop0, y_begin, y_end;
    int wrows, wy0;        // low-res rows of the weights, the first of them
    int strips, cblocks, segs, seg_rows;
};
// Work item: rows y0 .. y1 - 1 of a strip for one block of channels of one image; neighbouring strips run side by side.
struct Item { int n, c0, x0, y0, y1; };
template <typename T> __device__ __forceinline__ Item item_at(const SArgs &a, int i) {
    Item t;
    t.x0 = (i % a.strips) * Geo<T>::CELLS; i /= a.strips;
    t.y0 = a.y_begin + (i % a.segs) * a.seg_rows; i /= a.segs;
    t.y1 = min(t.y0 + a.seg_rows, a.y_end);
    t.c0 = (i % a.cblocks) * CH;
    t.n = i / a.cblocks;
    return t;
}

// One output over the cells of its own window alone; a NaN ends the sum.
template <typename T> __device__ __noinline__ float pixel_alone(const SArgs &a, int n, int c, int hy, int hx) {
    const size_t w_plane = (size_t)(2 * a.wrows) * (2 * a.W);
    const T *w = static_cast<const T *>(a.wt) + (size_t)n * 25 * w_plane + (size_t)(hy - 2 * a.wy0) * (2 * a.W) + hx;
    const T *v = static_cast<const T *>(a.v) + ((size_t)n * a.C + c) * a.rows * a.W;
    float s = 0.f;
#pragma unroll 1
    for (int k = 0; k < 25 && s == s; ++k) {
        const int y = a.ytop0 + (hy >> 1) + k / 5 - 2, x = (hx >> 1) + k % 5 - 2;
        if (y < 0 || y >= a.rows || x < 0 || x >= a.W) continue;
        const float wk = to_acc(w[k * w_plane]);
        s = wk == wk ? fmaf(wk, to_acc(v[(size_t)y * a.W + x]), s) : wk;
    }
    return s;
}
// Moves the cells of a product from a landed row, float32 in two terms; elements that are not finite become zeros and the row is noted.  The landed row is
// given back (`landed`) as soon as its values have been used: an arrival does not wait for loads in flight.
template <typename T>
__device__ __forceinline__ void move_cells(unsigned at, unsigned (&v)[4 * VCHUNKS], bool channel, finite::Noted &noted, int quarter, int row, unsigned landed) {
    using G = Geo<T>;
#pragma unroll
    for (int q = G::SHIFT + G::WORDS; q < G::SHIFT + ACOLS; ++q) v[q] = 0u;     // their weights are zero
    auto store = [&]() {
        tc_st16(at, v + G::SHIFT); tc_st8(at + 16, v + G::SHIFT + 16);          // the tensor core reads the top 19 bits of a tf32 operand
    };
    store();
    mbar_arrive(landed);
    const bool odd = !finite::all_finite<T, G::WORDS>(v + G::SHIFT);
    if (__any_sync(0xffffffffu, odd)) {
        tc_wait_st();
#pragma unroll
        for (int q = G::SHIFT; q < G::SHIFT + G::WORDS; ++q) v[q] = finite::or_zero<T>(v[q]);
        store();
        if (odd && channel) noted.note(quarter, row);                           // a lane without a channel holds anything
    }
    if constexpr (G::F32) {
#pragma unroll
        for (int q = G::SHIFT; q < G::SHIFT + ACOLS; ++q) v[q] = tf32_lo(v[q]);
        tc_st16(at + ACOLS, v + G::SHIFT); tc_st8(at + ACOLS + 16, v + G::SHIFT + 16);
    }
}
// Columns x0 - BOX0 and so on of value row dy of the step of low-res row y
template <typename T> __device__ __forceinline__ finite::Marks marks_of(const SArgs &a, int n, int c, int y, int dy, int x0) {
    finite::Marks m{0ull, 0ull, 0ull};
    const int row = a.ytop0 + y + dy - 2;
    if (row >= 0 && row < a.rows)
        finite::mark_row<T, (Geo<T>::CELLS + 2 * Geo<T>::BOX0) * (int)sizeof(T) / 16, false>(
            static_cast<const T *>(a.v) + (((size_t)n * a.C + c) * a.rows + row) * a.W, a.W, x0 - Geo<T>::BOX0, m);
    return m;
}
// Bits of parents (of the strip) whose windows hold a marked column
template <typename T> __device__ __forceinline__ unsigned long long reached(unsigned long long columns) {
    const unsigned long long m = columns >> (Geo<T>::BOX0 - 2);
    return (m | m >> 1 | m >> 2 | m >> 3 | m >> 4) & ((1ull << Geo<T>::CELLS) - 1);
}
// The pixels of a step and channel again, once they are stored, whose sums are not finite (sums: there may be such), or that have something not finite in
// their windows, which the product took as zero.  dy0, dy1: the window rows that may hold such elements.
template <typename T> __device__ __noinline__ void finish_pixels(const SArgs &a, int n, int c, int y, int x0, int dy0, int dy1, bool sums) {
    using G = Geo<T>;
    constexpr int FIRST = G::BOX0 - 2, PER = 16 / (int)sizeof(T);     // bit of a parent's first column; elements of 16 bytes
    constexpr unsigned long long ALL = (1ull << G::CELLS) - 1;
    unsigned long long nan = 0ull, up[5], down[5], any = 0ull;        // nan, any: parents with such an element in their windows
#pragma unroll 1
    for (int dy = 0; dy < 5; ++dy) {
        finite::Marks m{0ull, 0ull, 0ull};
        if (dy >= dy0 && dy <= dy1 && nan != ALL) m = marks_of<T>(a, n, c, y, dy, x0);
        nan |= reached<T>(m.nan); any |= reached<T>(m.any());
        up[dy] = m.up; down[dy] = m.down;
    }
    const size_t hi_plane = (size_t)(2 * a.H) * (2 * a.W), w_plane = (size_t)(2 * a.wrows) * (2 * a.W);
#pragma unroll 1
    for (int q = 0; q < 2 * G::PX / PER; ++q) {                       // chunks of 16 bytes of the two rows
        const int r = q / (G::PX / PER), px0 = q % (G::PX / PER) * PER;
        constexpr unsigned long long PARENTS = (1ull << PER / 2) - 1;
        if (x0 + px0 / 2 >= a.W || (!sums && (any >> px0 / 2 & PARENTS) == 0ull)) continue;
        const size_t at = (size_t)(2 * y + r) * (2 * a.W) + 2 * x0 + px0;
        T *const o = static_cast<T *>(a.out) + ((size_t)n * a.C + c) * hi_plane + at;
        if ((nan >> px0 / 2 & PARENTS) == PARENTS) {
            *reinterpret_cast<uint4 *>(o) = finite::nan_chunk<T>();
            continue;
        }
        const T *const wt = static_cast<const T *>(a.wt) + (size_t)n * 25 * w_plane + at - (size_t)(2 * a.wy0) * (2 * a.W);
        const uint4 w = __ldcg(reinterpret_cast<const uint4 *>(o));   // stored by TMA: not from L1
        const unsigned words[4] = {w.x, w.y, w.z, w.w};
        if (!finite::all_finite<T, 4>(words) && finite::all_nan<T>(*reinterpret_cast<const uint4 *>(wt + 12 * w_plane))) {
            *reinterpret_cast<uint4 *>(o) = finite::nan_chunk<T>();   // weights of NaN for the pixels' own cells
            continue;
        }
        float s[PER];                                                 // what the infinities alone come to
#pragma unroll
        for (int e = 0; e < PER; ++e) s[e] = 0.f;
#pragma unroll 1
        for (int k = 0; k < 25; ++k) {
            const unsigned u = (unsigned)(up[k / 5] >> (FIRST + px0 / 2 + k % 5)), d = (unsigned)(down[k / 5] >> (FIRST + px0 / 2 + k % 5));
            if (((u | d) & (unsigned)PARENTS) == 0u) continue;
            const uint4 wk = *reinterpret_cast<const uint4 *>(wt + k * w_plane);
#pragma unroll
            for (int e = 0; e < PER; ++e)
                if ((u | d) >> (e / 2) & 1) s[e] = fmaf(finite::element<T>(wk, e), u >> (e / 2) & 1 ? INFINITY : -INFINITY, s[e]);
        }
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int p = px0 / 2 + e / 2;
            if (!finite::is_finite<T>(words, e)) s[e] = pixel_alone<T>(a, n, c, 2 * y + r, 2 * x0 + px0 + e);
            else if ((any >> p & 1) == 0ull) continue;
            o[e] = from_acc<T>((nan >> p & 1) != 0ull ? finite::nan_value() : s[e]);
        }
    }
}
}  // namespace strip

template <typename T>
__global__ void __launch_bounds__(strip::NT, 1) sapa_strip_kernel(const __grid_constant__ CUtensorMap vmap, const __grid_constant__ CUtensorMap wmap,
                                                                  const __grid_constant__ CUtensorMap omap, const __grid_constant__ strip::SArgs a) {
    using namespace strip;
    using G = strip::Geo<T>;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * (NVL + NWL + strip::NV + ND + NP)];
    __shared__ unsigned tmem_slot;
    __shared__ finite::Noted noted;                                   // rows of V, counted over the CTA's items
    const unsigned base = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u;
    const unsigned vfull = (unsigned)__cvta_generic_to_shared(bars), vempty = vfull + 8 * NVL, wfull = vempty + 8 * NVL, wempty = wfull + 8 * NWL;
    const unsigned aready = wempty + 8 * NWL, aempty = aready + 8 * strip::NV, dfull = aempty + 8 * strip::NV, dempty = dfull + 8 * ND;
    const unsigned pready = dempty + 8 * ND, pempty = pready + 8 * NP;
    const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
    const int items = a.B * a.cblocks * a.segs * a.strips;

    if (tid < 4) noted.clear(tid);
    if (tid == 0) {
        for (int i = 0; i < NVL; ++i) { mbar_init(vfull + 8 * i, 1); mbar_init(vempty + 8 * i, 128); }
        for (int i = 0; i < NWL; ++i) { mbar_init(wfull + 8 * i, 1); mbar_init(wempty + 8 * i, 32 * P_WARPS); }
        for (int i = 0; i < strip::NV; ++i) { mbar_init(aready + 8 * i, 128); mbar_init(aempty + 8 * i, G::ISSUERS); }
        for (int i = 0; i < ND; ++i) { mbar_init(dfull + 8 * i, G::ISSUERS); mbar_init(dempty + 8 * i, 128); }
        for (int i = 0; i < NP; ++i) { mbar_init(pready + 8 * i, 32 * P_WARPS); mbar_init(pempty + 8 * i, G::ISSUERS); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == MMA_WARP) {
        tc_alloc((unsigned)__cvta_generic_to_shared(&tmem_slot), TMEM_COLS);
        tc_relinquish();
    }
    for (int i = tid; i < NP * G::P_BYTES / 16; i += strip::NT)
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(base + G::P0 + 16 * i), "r"(0u) : "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = warp_uniform(*reinterpret_cast<volatile unsigned *>(&tmem_slot));
    const unsigned quarter = (unsigned)((warp & 3) * 32) << 16;       // the lanes of tensor memory that a warp can reach
    const unsigned ring = ND * G::N;                                  // columns: accumulators, then the rows of V
    unsigned zeros[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) zeros[i] = 0u;
    if (warp < EPI_WARPS) {
#pragma unroll 1
        for (int c = 0; c < G::N; c += 16) tc_st16(tmem + quarter + (warp >> 2) * G::N + c, zeros);
        tc_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    begin_after_previous();

    bool ok = true;
    if (warp == TMA_WARP) {
        if (lane == 0) {
            int vs = 0, vph = 0, ws = 0, wph = 0;
            const int vbytes = min(a.C, CH) * VROW;
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item t = item_at<T>(a, i);
                for (int y = t.y0 - 2; y < t.y1 + 2 && ok; ++y) {     // the row of V, and the weights of the pixels it completes the windows of
                    if (!mbar_wait_bounded(vempty + 8 * vs, vph ^ 1)) { ok = false; break; }
                    mbar_expect_tx(vfull + 8 * vs, vbytes);
                    tma_load_4d(base + G::V0 + vs * strip::V_BYTES, &vmap, vfull + 8 * vs, t.x0 - G::BOX0, t.c0, a.ytop0 + y, t.n);
                    if (++vs == NVL) { vs = 0; vph ^= 1; }
                    if (y < t.y0 + 2) continue;
                    if (!mbar_wait_bounded(wempty + 8 * ws, wph ^ 1)) { ok = false; break; }
                    mbar_expect_tx(wfull + 8 * ws, L_BYTES);
                    tma_load_4d(base + G::L0 + ws * L_BYTES, &wmap, wfull + 8 * ws, 2 * t.x0, 0, 2 * (y - 2 - a.wy0), t.n);
                    if (++ws == NWL) { ws = 0; wph ^= 1; }
                }
            }
            if (!ok) {                                                // none of its loads may land after it has left
                (void)drain_loads<NVL>(vfull, vs, vph);
                (void)drain_loads<NWL>(wfull, ws, wph);
            }
        }
    } else if (warp >= MMA_WARP) {
        constexpr unsigned HI = (128u >> 4) | (1u << 14);             // 8-row groups 128 bytes apart, descriptor version 1, no swizzle
        const unsigned leader = elect_leader(), p_base = warp_uniform(base + G::P0);
        const unsigned b0 = desc_lo(p_base + G::tile(0), G::lbo(0)), b1 = desc_lo(p_base + G::tile(1), G::lbo(1)), b2 = desc_lo(p_base + G::tile(2), G::lbo(2));
        // the products of a tile that reach parents [lo, hi) of the strip; nothing where there are none
        auto part = [&](auto tile, auto lo, auto hi, unsigned d, unsigned ka, unsigned b) {
            constexpr int J = decltype(tile)::value, LO = decltype(lo)::value, HI_P = decltype(hi)::value;
            constexpr int P = (LO > G::p0(J)) ? LO : G::p0(J), ROWS = 4 * (((HI_P < G::p1(J)) ? HI_P : G::p1(J)) - P);
            if constexpr (ROWS > 0) tc_mma_ta<G::F32>(leader, d + 4 * P, ka + 8 * J, b + 4 * (P - G::p0(J)), HI, IDESC_M128<T> | idesc_n(ROWS), 1u);
        };
        int row0 = 0, db = 0, dph = 0, pb = 0, pph = 0;               // row0: rows of V of this CTA before the item
        auto run = [&](auto lo, auto hi) {
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item t = item_at<T>(a, i);
                int known = row0;                                     // rows of V waited for
                for (int s = 0; s < t.y1 - t.y0 && ok; ++s) {
                    for (; known < row0 + s + 5 && ok; ++known) ok = mbar_wait_warp(aready + 8 * (known % strip::NV), (known / strip::NV) & 1);
                    ok = ok && mbar_wait_warp(dempty + 8 * db, dph ^ 1) && mbar_wait_warp(pready + 8 * pb, pph);
                    if (!ok) break;
                    tc_fence_after();
                    const unsigned d = tmem + db * G::N, pofs = (unsigned)(pb * G::P_BYTES) >> 4;
                    auto product = [&](int av, int pt) {              // terms of V and of P
#pragma unroll
                        for (int dy = 0; dy < 5; ++dy) {
                            const unsigned ka = tmem + ring + ((row0 + s + dy) % strip::NV) * G::ABUF + av * ACOLS;
                            const unsigned kb = pofs + ((dy * G::DY_BYTES + pt * G::P_TERM) >> 4);
                            part(std::integral_constant<int, 0>{}, lo, hi, d, ka, b0 + kb);
                            part(std::integral_constant<int, 1>{}, lo, hi, d, ka, b1 + kb);
                            part(std::integral_constant<int, 2>{}, lo, hi, d, ka, b2 + kb);
                        }
                    };
                    if (G::F32) { product(1, 0); product(0, 1); }
                    product(0, 0);
                    tc_commit_by(leader, dfull + 8 * db);
                    tc_commit_by(leader, pempty + 8 * pb);
                    tc_commit_by(leader, aempty + 8 * ((row0 + s) % strip::NV));
                    if (++db == ND) { db = 0; dph ^= 1; }
                    if (++pb == NP) { pb = 0; pph ^= 1; }
                }
                row0 += t.y1 - t.y0;
                if (ok)
                    for (int q = 0; q < 4; ++q) tc_commit_by(leader, aempty + 8 * ((row0 + q) % strip::NV));   // the last step's other rows
                row0 += 4;
            }
        };
        constexpr int HALF = G::CELLS / G::ISSUERS;
        if (warp == MMA_WARP) run(std::integral_constant<int, 0>{}, std::integral_constant<int, HALF>{});
        else if (G::ISSUERS == 2) run(std::integral_constant<int, HALF>{}, std::integral_constant<int, G::CELLS>{});
    } else if (warp >= SPLIT_WARP0 && warp < P_WARP0) {
        int vs = 0, vph = 0, as = 0, aph = 0, row = 0;
        const unsigned line = ((warp & 3) * 32 + lane) * VROW;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = item_at<T>(a, i);
            const bool used = t.c0 + (warp & 3) * 32 < a.C;           // lanes without a channel keep whatever they hold
            for (int y = t.y0 - 2; y < t.y1 + 2; ++y, ++row) {
                if (!mbar_wait_warp(vfull + 8 * vs, vph)) { ok = false; break; }
                unsigned v[4 * VCHUNKS];
                if (used) {
#pragma unroll
                    for (int q = 0; q < G::LOADS; ++q)
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[4 * q]), "=r"(v[4 * q + 1]), "=r"(v[4 * q + 2]), "=r"(v[4 * q + 3])
                                     : "r"(base + G::V0 + vs * strip::V_BYTES + line + 16 * q) : "memory");
                }
                if (!mbar_wait_warp(aempty + 8 * as, aph ^ 1)) { ok = false; break; }
                tc_fence_after();
                if (used) move_cells<T>(tmem + quarter + ring + as * G::ABUF, v, t.c0 + (warp & 3) * 32 + lane < a.C, noted, warp & 3, row, vempty + 8 * vs);
                else mbar_arrive(vempty + 8 * vs);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(aready + 8 * as);
                if (++vs == NVL) { vs = 0; vph ^= 1; }
                if (++as == strip::NV) { as = 0; aph ^= 1; }
            }
        }
    } else if (warp >= P_WARP0 && warp < TMA_WARP) {
        // A unit: window row dy for 32 pixels, 16 of each high-res row (columns 16 q ..) in 16 bits, 32 of one row in float32; a lane holds the five
        // weights of a pixel's window row and writes them to its cells.
        constexpr int Q = G::N / 32, UNITS = 5 * Q, NU = (UNITS + P_WARPS - 1) / P_WARPS, ST = G::F32 ? 5 : 3;
        int from[NU], to[NU][ST];
        bool odd = false;
#pragma unroll
        for (int i = 0; i < NU; ++i) {
            const int unit = i * P_WARPS + warp - P_WARP0, dy = unit / Q, q = unit % Q;
            const int r = G::F32 ? q & 1 : lane >> 4, px = G::F32 ? 32 * (q >> 1) + lane : 16 * q + (lane & 15), parent = px >> 1, n = 4 * parent + 2 * r + (px & 1);
            from[i] = unit < UNITS ? (r * 25 + dy * 5) * 128 + px * (int)sizeof(T) : -1;
            odd = parent & 1;
#pragma unroll
            for (int e = 0; e < ST; ++e) to[i][e] = dy * G::DY_BYTES + (G::F32 ? G::at(n, parent + e) : G::at(n, (parent & ~1) + 2 * e));
        }
        int ws = 0, wph = 0, pb = 0, pph = 0;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = item_at<T>(a, i);
            for (int y = t.y0; y < t.y1; ++y) {
                if (!mbar_wait_bounded(wfull + 8 * ws, wph)) { ok = false; break; }
                const unsigned src = fresh(base + G::L0 + ws * L_BYTES), dst = base + G::P0 + pb * G::P_BYTES;
                unsigned w[NU][5];
#pragma unroll
                for (int u = 0; u < NU; ++u)
                    if (from[u] >= 0)
#pragma unroll
                        for (int dx = 0; dx < 5; ++dx) {
                            if constexpr (G::F32) {
                                w[u][dx] = lds32(src + from[u] + 128 * dx);
                            } else {
                                unsigned short x;
                                asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(x) : "r"(src + from[u] + 128 * dx) : "memory");
                                w[u][dx] = x;
                            }
                        }
                if (!mbar_wait_bounded(pempty + 8 * pb, pph ^ 1)) { ok = false; break; }
#pragma unroll
                for (int u = 0; u < NU; ++u)
                    if (from[u] >= 0) {
                        if constexpr (G::F32) {
#pragma unroll
                            for (int dx = 0; dx < 5; ++dx) {
                                sts32(dst + to[u][dx], w[u][dx]);
                                sts32(dst + G::P_TERM + to[u][dx], tf32_lo(w[u][dx]));
                            }
                        } else {                                      // cell pairs start at even cells
                            sts32(dst + to[u][0], odd ? w[u][0] << 16 : w[u][0] | w[u][1] << 16);
                            sts32(dst + to[u][G::F32 ? 0 : 1], odd ? w[u][1] | w[u][2] << 16 : w[u][2] | w[u][3] << 16);
                            sts32(dst + to[u][G::F32 ? 0 : 2], odd ? w[u][3] | w[u][4] << 16 : w[u][4]);
                        }
                    }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                mbar_arrive(pready + 8 * pb);
                mbar_arrive(wempty + 8 * ws);
                if (++ws == NWL) { ws = 0; wph ^= 1; }
                if (++pb == NP) { pb = 0; pph ^= 1; }
            }
        }
    } else if (warp < EPI_WARPS) {
        const int group = warp >> 2;                                  // a warpgroup for each accumulator: every second step
        const unsigned box = base + G::OUT0 + warp * OUT_BYTES, stage = box + lane * 128, d = tmem + quarter + group * G::N;
        int step = 0, dph = 0, row0 = 0;                              // row0: rows of V of this CTA before the item
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = item_at<T>(a, i);
            const int cw = t.c0 + (warp & 3) * 32, c = cw + lane;
            for (int y = t.y0; y < t.y1; ++y, ++step) {
                if ((step & 1) != group) continue;
                if (!mbar_wait_warp(dfull + 8 * group, dph)) { ok = false; break; }
                dph ^= 1;
                tc_fence_after();
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");       // the last store has read the box
                __syncwarp();
                float zero[4] = {0.f, 0.f, 0.f, 0.f};                 // stays zero while all values are finite
#pragma unroll
                for (int g = 0; g < G::N / 32; ++g) {                 // 8 parents at a time: 16 pixels of both high-res rows
                    unsigned v[32];
                    tc_ld16(d + 32 * g, *reinterpret_cast<unsigned (*)[16]>(&v[0]));
                    tc_ld16(d + 32 * g + 16, *reinterpret_cast<unsigned (*)[16]>(&v[16]));
                    tc_wait_ld();
                    tc_st16(d + 32 * g, zeros);
                    tc_st16(d + 32 * g + 16, zeros);
#pragma unroll
                    for (int e = 0; e < 32; ++e) zero[e & 3] = fmaf(__uint_as_float(v[e]), 0.f, zero[e & 3]);
                    constexpr int PER = 16 / (int)sizeof(T);          // pixels of a chunk
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int q = 0; q < 16 / PER; ++q) {
                            auto px = [&](int e) { return v[4 * ((q * PER + e) >> 1) + 2 * r + (e & 1)]; };
                            uint4 w;
                            if constexpr (G::F32) {
                                w = make_uint4(px(0), px(1), px(2), px(3));
                            } else {
                                w.x = pack_pair(T(), __uint_as_float(px(0)), __uint_as_float(px(1)));
                                w.y = pack_pair(T(), __uint_as_float(px(2)), __uint_as_float(px(3)));
                                w.z = pack_pair(T(), __uint_as_float(px(4)), __uint_as_float(px(5)));
                                w.w = pack_pair(T(), __uint_as_float(px(6)), __uint_as_float(px(7)));
                            }
                            const int chunk = g * (16 / PER) + q;
                            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(stage + r * (32 * 128) + ((chunk ^ (lane & 7)) << 4)),
                                         "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
                        }
                }
                if (!((zero[0] + zero[1]) + (zero[2] + zero[3]) == 0.f) && c < a.C) noted.note_sum(warp & 3, row0 + y - t.y0);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(dempty + 8 * group);
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0 && cw < a.C) {                          // pixels and channels beyond the tensor are cut off
                    tma_store_4d(&omap, box, 2 * t.x0, cw, 2 * y, t.n);
                    tma_store_4d(&omap, box + 32 * 128, 2 * t.x0, cw, 2 * y + 1, t.n);
                    asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                }
            }
            row0 += t.y1 - t.y0 + 4;
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
    if (!ok) atomicExch(&g_wait_timeout, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == MMA_WARP) tc_dealloc(tmem, TMEM_COLS);
    if (warp < EPI_WARPS && noted.last[warp & 3] >= 0) {              // rare: outputs with something not finite (all are stored)
        const int first = noted.first[warp & 3], last = noted.last[warp & 3];
        int row = 0;
        for (int i = blockIdx.x; i < items; i += gridDim.x, row += 4) {
            const Item t = item_at<T>(a, i);
            const int c = t.c0 + (warp & 3) * 32 + lane;
            for (int y = t.y0; y < t.y1; ++y, ++row)
                if ((y & 1) == warp >> 2 && c < a.C && row + 4 >= first && row <= last)
                    finish_pixels<T>(a, t.n, c, y, t.x0, first - row, last - row, noted.sums[warp & 3] != 0);
        }
    }
}
