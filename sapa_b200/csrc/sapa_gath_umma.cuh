// sapa_gath_umma.cuh — the transposed aggregation of sapa_gath_mma.cu on the 5th-generation tensor cores (included there), for rows
// of 16 bytes:
//
//     G[c][u] = sum over high-res pixels p and window slots k with win_k(p) = u of  X[c][p] * Wt[k][p]
//
// A CTA walks strips of low-res columns (16 in float32, 32 in 16 bits) down the image, one high-res row of 128 channels at a time.
// For one high-res row, all output rows that it reaches (its parent's five) are ONE product
//     D[128 ch x (5 rows x strip)] += X[128 ch x K px] * W[K px x (5 rows x strip)],     K px = 40 (float32) or 80
// in tensor memory, where the strip's output rows form a ring of slots: a row of the ring is opened four parent rows before it is
// complete, and drained while later ones accumulate.
//   * X: one TMA box (128 channels x 176 bytes of one high-res row; rows of an odd number of 16-byte chunks are read without
//     bank conflicts) per step, with the same pixels of the 25 weight planes behind it.  Two warpgroups take turns to move a landed box
//     into tensor memory as the A operand (lane = channel, column = 32 bits of pixels); float32 is split on the way, once per element,
//     into the two tf32 terms of the three-term product (hi*hi + lo*hi + hi*lo).
//   * W: the operand [5 x strip rows][K px] of a step is banded, and its zeros are the same in every step: they are written once,
//     and two warpgroups in turn overwrite the 25 weights per pixel that are not zero (unswizzled 8 x 16 byte core matrices, the leading
//     offset padded by 16 bytes so that the stores of a warp spread over the banks).
//   * one warp issues the MMAs: 15 (float32) or 5 per step, of N = 80 or 160, at N / 2 clocks each (tc_mma_ta).
//   * float32 keeps three sums per output (hi*hi of the upper and of the lower high-res rows, and the small products), which the epilogue adds:
//     an accumulation in tensor memory rounds toward zero, and one sum of all sixty is 1.5e-6 from float64, these three 5.1e-7 (the
//     kernel on tiles 5.3e-7).
//   * epilogue: tcgen05.ld (lane = channel), 16-byte stores, and zeros back into the slot.
//   * what is not finite stays out of the products (finite.cuh); a second pass forms the cells that it reaches.
// The mma.sync kernel of sapa_gath_mma.cu splits and loads an element once per output row that it reaches and is bound by that.  What
// bounds this one: no unit alone.  8 x 256 x 64x64, value gradient, under ncu: tensor pipe 46 % of the time in float32, 30 % in 16 bits, memory 40 and 34 %,
// shared-memory loads and stores of the warps 25 and 21 %; a step's box is landed, moved and multiplied one behind the other, and in 16 bits a strip's boxes
// hold 1.4 times its pixels.  float32 104 -> 45 us (4.0 TB/s), bfloat16 43 -> 24 (3.7 TB/s).
// Every wait is bounded and raises g_wait_timeout; a CTA that gives up drains its loads and frees its tensor memory.

namespace gumma {

using namespace ummau;

constexpr int CH = 128;                                     // channels of a step = lanes of tensor memory
constexpr int MAX_NX = 8, NWB = 4;                          // steps of X in flight (as many as fit the ring, an even number), of W
                                                            // (even: a warpgroup that takes every second step has slots of its own)
constexpr int SPLIT_WARPS = 8, EPI_WARP0 = 8, W_WARP0 = 12, TMA_WARP = 20, MMA_WARP = 21, NT = 22 * 32;
constexpr int XROW = 176, XCHUNKS = 10;                     // bytes of a box row; 16-byte chunks of it that the product reads
constexpr int L_BYTES = 25 * XROW;                          // of a step: the pixels of its box in the 25 weight planes
constexpr int RING_BYTES = 4 * ((CH * XROW + L_BYTES + 127) / 128 * 128);
constexpr int ACOLS = 4 * XCHUNKS;                          // columns of an A operand (one term)
constexpr int TMEM_COLS = 512;

template <typename T> struct Geo {
    static constexpr bool F32 = sizeof(T) == 4;
    static constexpr int CELLS = F32 ? 16 : 32;             // low-res columns of a strip
    static constexpr int P0 = F32 ? 2 : 4;                  // the box starts at the pixels of parent x0 - P0 (a 16-byte boundary)
    static constexpr int KSTEPS = 5;                        // of 32 bytes
    static constexpr int N = 5 * CELLS;
    static constexpr int TERMS = F32 ? 2 : 1, SUMS = F32 ? 3 : 1;
    static constexpr int SLOTS = F32 ? 7 : 8;               // output rows in tensor memory: five that accumulate, the rest being drained
    static constexpr int DSUM = SLOTS * CELLS;              // columns from one kind of sum to the next
    static constexpr int DCOLS = SUMS * DSUM;
    static constexpr int ABUF = TERMS * ACOLS, NA = F32 ? 2 : 6;
    static constexpr int LBO = N * 16 + 16, W_TERM = XCHUNKS * LBO, W_BYTES = TERMS * W_TERM;
    static constexpr int PP = CELLS + 4;                    // parents whose windows reach the strip
    static constexpr int ITEMS = 25 * PP, NI = (ITEMS + 127) / 128;
    static constexpr int SMEM = RING_BYTES + NWB * W_BYTES + 1024;
    static_assert(DCOLS % 16 == 0 && DCOLS + NA * ABUF <= TMEM_COLS, "tensor memory");
};

struct UArgs {
    Args g;
    int strips, cblocks, segs, seg_rows;
    int nx, x_bytes, slot_bytes;                            // ring: slots; bytes of a slot's box of X, of the whole slot
};

// Work item: a strip's rows y0 .. y1 - 1 for one block of channels of one image.  Neighbouring strips run side by side, because
// their boxes overlap.
struct Item { int n, c0, x0, y0, y1; };
template <typename T> __device__ __forceinline__ Item item_at(const UArgs &u, int i) {
    Item t;
    t.x0 = (i % u.strips) * Geo<T>::CELLS; i /= u.strips;
    t.y0 = (i % u.segs) * u.seg_rows; i /= u.segs;
    t.y1 = min(t.y0 + u.seg_rows, u.g.Hout);
    t.c0 = (i % u.cblocks) * CH;
    t.n = i / u.cblocks;
    return t;
}
// the parent rows (of the frame of the high-res rows) that reach an item, clipped to the image
__device__ __forceinline__ int first_parent(const UArgs &u, const Item &t) { return max(t.y0 - u.g.top - 2, 0); }
// (none for an item of rows that the slab's pixels do not reach)
__device__ __forceinline__ int end_parent(const UArgs &u, const Item &t) { return max(min(t.y1 - u.g.top + 2, u.g.H), first_parent(u, t)); }

// Parents of strip columns x0 - P0 and so on that hold something not finite in high-res row h of channel c
template <typename T> __device__ __forceinline__ finite::Marks marks_of(const Args &a, int n, int c, int h, int x0) {
    finite::Marks m{0ull, 0ull, 0ull};
    finite::mark_row<T, XCHUNKS, true>(static_cast<const T *>(a.hi) + (((size_t)n * a.C + c) * (2 * a.H) + h) * (2 * a.W), 2 * a.W, 2 * (x0 - Geo<T>::P0), m);
    return m;
}
// The cells of a strip's output row and channel again whose sums are not finite (sums: there may be such), or that high-res rows ha .. hb - 1 reach with something not finite, which
// the product took as zero: over their own pixels alone.
template <typename T> __device__ __noinline__ void finish_cells(const UArgs &u, int n, int c, int y, int x0, int ha, int hb, bool sums) {
    using G = Geo<T>;
    const Args &a = u.g;
    auto reached = [](unsigned long long parents) {                   // bits of cells of the strip
        const unsigned long long m = parents >> (G::P0 - 2);
        return (unsigned)((m | m >> 1 | m >> 2 | m >> 3 | m >> 4) & ((1ull << G::CELLS) - 1));
    };
    constexpr unsigned ALL = (unsigned)((1ull << G::CELLS) - 1);
    unsigned nan = 0u, any = 0u;                                      // cells that a NaN, that something not finite reaches
#pragma unroll 1
    for (int h = ha; h < hb && nan != ALL; ++h) {
        const finite::Marks m = marks_of<T>(a, n, c, h, x0);
        nan |= reached(m.nan); any |= reached(m.any());
    }
    T *const o = static_cast<T *>(a.out) + (((size_t)n * a.C + c) * a.Hout + y) * a.W + x0;
    constexpr int PER = 16 / (int)sizeof(T);
    constexpr unsigned CHUNK = (1u << PER) - 1;
#pragma unroll 1
    for (int q0 = 0; q0 < G::CELLS && x0 + q0 < a.W; q0 += PER) {
        if (!sums && (any >> q0 & CHUNK) == 0u) continue;
        if ((nan >> q0 & CHUNK) == CHUNK) {
            *reinterpret_cast<uint4 *>(o + q0) = finite::nan_chunk<T>();
            continue;
        }
        const int yp = y - a.top;
        if (yp >= 0 && yp < a.H) {                                    // weights of NaN of the cells' own parents
            const T *w = static_cast<const T *>(a.wt) + (((size_t)n * 25 + 12) * (2 * a.H) + 2 * yp) * (2 * a.W) + 2 * (x0 + q0);
            if (finite::all_nan<T>(*reinterpret_cast<const uint4 *>(w)) && finite::all_nan<T>(*reinterpret_cast<const uint4 *>(w + PER))) {
                *reinterpret_cast<uint4 *>(o + q0) = finite::nan_chunk<T>();
                continue;
            }
        }
#pragma unroll 1
        for (int q = q0; q < q0 + PER; ++q)
            if ((any >> q & 1) != 0u || !isfinite(to_acc(o[q]))) o[q] = from_acc<T>(nan >> q & 1 ? finite::nan_value() : cell_sum<T>(a, n, c, y, x0 + q));
    }
}

template <typename T>
__global__ void __launch_bounds__(NT, 1) sapa_gath_umma_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap lmap, const __grid_constant__ UArgs u) {
    using G = Geo<T>;
    const Args &a = u.g;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) unsigned long long bars[2 * MAX_NX + 2 * NWB + 2 * G::NA + 2 * G::SLOTS];
    __shared__ unsigned tmem_slot;
    __shared__ finite::Noted noted;                                   // steps, counted over the CTA's items
    const unsigned ring = ((unsigned)__cvta_generic_to_shared(smem_dyn) + 1023u) & ~1023u, wbuf = ring + RING_BYTES;
    const unsigned xfull = (unsigned)__cvta_generic_to_shared(bars), xempty = xfull + 8 * MAX_NX;
    const unsigned wready = xempty + 8 * MAX_NX, wempty = wready + 8 * NWB, aready = wempty + 8 * NWB, aempty = aready + 8 * G::NA;
    const unsigned dfull = aempty + 8 * G::NA, dempty = dfull + 8 * G::SLOTS;
    const int tid = threadIdx.x, warp = (int)warp_uniform(tid >> 5), lane = tid & 31;
    const int items = a.B * u.cblocks * u.segs * u.strips;

    if (tid < 4) noted.clear(tid);
    if (tid == 0) {
        for (int i = 0; i < u.nx; ++i) { mbar_init(xfull + 8 * i, 1); mbar_init(xempty + 8 * i, 256); }
        for (int i = 0; i < NWB; ++i) { mbar_init(wready + 8 * i, 128); mbar_init(wempty + 8 * i, 1); }
        for (int i = 0; i < G::NA; ++i) { mbar_init(aready + 8 * i, 128); mbar_init(aempty + 8 * i, 1); }
        for (int i = 0; i < G::SLOTS; ++i) { mbar_init(dfull + 8 * i, 1); mbar_init(dempty + 8 * i, 128); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == MMA_WARP) {
        tc_alloc((unsigned)__cvta_generic_to_shared(&tmem_slot), TMEM_COLS);
        tc_relinquish();
    }
    for (int i = tid; i < NWB * G::W_BYTES / 16; i += NT)
        asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(wbuf + 16 * i), "r"(0u) : "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = warp_uniform(*reinterpret_cast<volatile unsigned *>(&tmem_slot));
    const unsigned quarter = (unsigned)((warp & 3) * 32) << 16;       // the lanes of tensor memory that a warp can reach
    unsigned zeros[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) zeros[i] = 0u;
    if (warp >= EPI_WARP0 && warp < W_WARP0) {
#pragma unroll 1
        for (int c = 0; c < G::DCOLS; c += 16) tc_st16(tmem + quarter + c, zeros);
        tc_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    begin_after_previous();

    bool ok = true;
    if (warp == TMA_WARP) {
        if (lane == 0) {
            int slot = 0, phase = 0;
            const int bytes = min(a.C, CH) * XROW + L_BYTES;          // of the boxes, zeros outside the tensors included
            for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
                const Item t = item_at<T>(u, i);
                for (int h = 2 * first_parent(u, t), he = 2 * end_parent(u, t); h < he; ++h) {
                    if (!mbar_wait_bounded(xempty + 8 * slot, phase ^ 1)) { ok = false; break; }
                    mbar_expect_tx(xfull + 8 * slot, bytes);
                    tma_load_4d(ring + slot * u.slot_bytes, &xmap, xfull + 8 * slot, 2 * (t.x0 - G::P0), t.c0, h, t.n);
                    tma_load_4d(ring + slot * u.slot_bytes + u.x_bytes, &lmap, xfull + 8 * slot, 2 * (t.x0 - G::P0), 0, h, t.n);
                    if (++slot == u.nx) { slot = 0; phase ^= 1; }
                }
            }
            if (!ok)                                                  // none of its loads may land after it has left
                for (int i = 0; i < u.nx; ++i) (void)mbar_wait_bounded(xfull + 8 * i, i < slot ? phase : phase ^ 1);
        }
    } else if (warp == MMA_WARP) {
        constexpr unsigned HI = (128u >> 4) | (1u << 14);             // 8-row groups 128 bytes apart, descriptor version 1, no swizzle
        const unsigned b_base = warp_uniform(desc_lo(wbuf, G::LBO)), leader = elect_leader();
        int ab = 0, aph = 0, wb = 0, wph = 0, cr0 = 0;                // cr0: output rows of this CTA before the item
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = item_at<T>(u, i);
            int opened = t.y0;
            for (int r = t.y0 - a.top - 2; r < t.y1 - a.top + 2 && ok; ++r) {
                const int u0 = r + a.top - 2;                         // output row of window row 0
                for (; opened < min(u0 + 5, t.y1) && ok; ++opened) {
                    const int cr = cr0 + opened - t.y0;
                    ok = mbar_wait_warp(dempty + 8 * (cr % G::SLOTS), ((cr / G::SLOTS) & 1) ^ 1);
                }
                if (ok && r >= 0 && r < a.H) {
                    const int j0 = max(0, t.y0 - u0), j1 = min(5, t.y1 - u0), s0 = (cr0 + u0 + j0 - t.y0) % G::SLOTS;
                    const int n1 = min(j1 - j0, G::SLOTS - s0), n2 = j1 - j0 - n1;          // window rows before the ring's end, behind it
                    const unsigned d1 = tmem + s0 * G::CELLS, i1 = IDESC_M128<T> | idesc_n(n1 * G::CELLS), i2 = IDESC_M128<T> | idesc_n(n2 * G::CELLS);
                    for (int e = 0; e < 2 && ok; ++e) {
                        ok = mbar_wait_warp(aready + 8 * ab, aph) && mbar_wait_warp(wready + 8 * wb, wph);
                        if (!ok) break;
                        tc_fence_after();
                        const unsigned at = tmem + G::DCOLS + ab * G::ABUF, b1 = b_base + ((wb * G::W_BYTES + j0 * G::CELLS * 16) >> 4);
                        auto product = [&](unsigned d, unsigned b, unsigned idesc) {
#pragma unroll
                            for (int ks = 0; ks < G::KSTEPS; ++ks) {
                                const unsigned ka = at + 8 * ks, kb = b + ks * (2 * G::LBO >> 4);
                                tc_mma_ta<G::F32>(leader, d + (G::F32 ? e * G::DSUM : 0), ka, kb, HI, idesc, 1u);
                                if (G::F32) {
                                    tc_mma_ta<G::F32>(leader, d + 2 * G::DSUM, ka + ACOLS, kb, HI, idesc, 1u);
                                    tc_mma_ta<G::F32>(leader, d + 2 * G::DSUM, ka, kb + (G::W_TERM >> 4), HI, idesc, 1u);
                                }
                            }
                        };
                        product(d1, b1, i1);
                        if (n2 > 0) product(tmem, b1 + ((n1 * G::CELLS * 16) >> 4), i2);
                        tc_commit_by(leader, aempty + 8 * ab);
                        tc_commit_by(leader, wempty + 8 * wb);
                        if (++ab == G::NA) { ab = 0; aph ^= 1; }
                        if (++wb == NWB) { wb = 0; wph ^= 1; }
                    }
                }
                if (ok && u0 >= t.y0 && u0 < t.y1) tc_commit_by(leader, dfull + 8 * ((cr0 + u0 - t.y0) % G::SLOTS));   // no later parent reaches this row
            }
            cr0 += t.y1 - t.y0;
        }
    } else if (warp < SPLIT_WARPS) {
        const int group = warp >> 2;                                  // takes every second step
        int slot = 0, phase = 0, ab = 0, aph = 0, step = 0;
        const unsigned row = ((warp & 3) * 32 + lane) * XROW;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = item_at<T>(u, i);
            for (int h = 2 * first_parent(u, t), he = 2 * end_parent(u, t); h < he; ++h, ++step) {
                if ((step & 1) == group) {
                    if (!mbar_wait_warp(xfull + 8 * slot, phase)) { ok = false; break; }
                    unsigned v[ACOLS];
                    if (t.c0 + (warp & 3) * 32 < a.C) {               // lanes without a channel keep whatever they hold
#pragma unroll
                        for (int q = 0; q < XCHUNKS; ++q)
                            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v[4 * q]), "=r"(v[4 * q + 1]), "=r"(v[4 * q + 2]), "=r"(v[4 * q + 3])
                                         : "r"(ring + slot * u.slot_bytes + row + 16 * q) : "memory");
                    }
                    if (!mbar_wait_warp(aempty + 8 * ab, aph ^ 1)) { ok = false; break; }
                    tc_fence_after();
                    if (t.c0 + (warp & 3) * 32 < a.C) {
                        const unsigned at = tmem + quarter + G::DCOLS + ab * G::ABUF;
                        auto store = [&]() { tc_st16(at, v); tc_st16(at + 16, v + 16); tc_st8(at + 32, v + 32); };      // the tensor core reads the top 19 bits of a tf32 operand
                        store();
                        mbar_arrive(xempty + 8 * slot);               // only here: an arrival does not wait for loads in flight
                        const bool odd = !finite::all_finite<T, ACOLS>(v);
                        if (__any_sync(0xffffffffu, odd)) {
                            tc_wait_st();
#pragma unroll
                            for (int q = 0; q < ACOLS; ++q) v[q] = finite::or_zero<T>(v[q]);
                            store();
                            if (odd && t.c0 + (warp & 3) * 32 + lane < a.C) noted.note(warp & 3, step);
                        }
                        if constexpr (G::F32) {
#pragma unroll
                            for (int q = 0; q < ACOLS; ++q) v[q] = tf32_lo(v[q]);
                            tc_st16(at + ACOLS, v); tc_st16(at + ACOLS + 16, v + 16); tc_st8(at + ACOLS + 32, v + 32);
                        }
                    } else {
                        mbar_arrive(xempty + 8 * slot);
                    }
                    tc_wait_st();
                    tc_fence_before();
                    mbar_arrive(aready + 8 * ab);
                }
                if (++slot == u.nx) { slot = 0; phase ^= 1; }
                if (++ab == G::NA) { ab = 0; aph ^= 1; }
            }
        }
    } else if (warp >= W_WARP0 && warp < TMA_WARP) {
        // An item: the pixel pair of parent pi (strip coordinate pi - 2) in window slot (dy, dx): operand row dy * strip + (pi + dx - 4),
        // pixels k, k + 1.  Pairs whose cell lies outside the strip are left out.
        const int wt = (tid - W_WARP0 * 32) & 127, group = (warp - W_WARP0) >> 2;      // two warpgroups take turns
        int from[G::NI], to[G::NI];
#pragma unroll
        for (int i = 0; i < G::NI; ++i) {
            const int idx = i * 128 + wt, k = idx / G::PP, pi = idx % G::PP, c = pi + k % 5 - 4, px = 2 * (G::P0 - 2 + pi);
            const int n = (k / 5) * G::CELLS + c;
            constexpr int PC = 16 / (int)sizeof(T);                   // pixels of a 16-byte chunk
            to[i] = idx < G::ITEMS && c >= 0 && c < G::CELLS ? (px / PC) * G::LBO + n * 16 + (px % PC) * (int)sizeof(T) : -1;
            from[i] = u.x_bytes + (idx < G::ITEMS ? k * XROW + px * (int)sizeof(T) : 0);
        }
        int slot = 0, phase = 0, wb = 0, wph = 0, step = 0;
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = item_at<T>(u, i);
            for (int h = 2 * first_parent(u, t), he = 2 * end_parent(u, t); h < he; ++h, ++step) {
                if ((step & 1) == group) {
                    if (!mbar_wait_bounded(xfull + 8 * slot, phase)) { ok = false; break; }
                    const unsigned src = fresh(ring + slot * u.slot_bytes), dst = wbuf + wb * G::W_BYTES;
                    unsigned v[G::NI][G::F32 ? 2 : 1];
#pragma unroll
                    for (int q = 0; q < G::NI; ++q) {
                        v[q][0] = lds32(src + from[q]);
                        if (G::F32) v[q][G::F32 ? 1 : 0] = lds32(src + from[q] + 4);
                    }
                    if (!mbar_wait_bounded(wempty + 8 * wb, wph ^ 1)) { ok = false; break; }
#pragma unroll
                    for (int q = 0; q < G::NI; ++q)
                        if (to[q] >= 0) {
                            if constexpr (G::F32) {
                                sts64(dst + to[q], __uint_as_float(v[q][0]), __uint_as_float(v[q][1]));
                                sts64(dst + G::W_TERM + to[q], __uint_as_float(tf32_lo(v[q][0])), __uint_as_float(tf32_lo(v[q][1])));
                            } else {
                                sts32(dst + to[q], v[q][0]);
                            }
                        }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    mbar_arrive(wready + 8 * wb);
                    mbar_arrive(xempty + 8 * slot);
                }
                if (++slot == u.nx) { slot = 0; phase ^= 1; }
                if (++wb == NWB) { wb = 0; wph ^= 1; }
            }
        }
    } else {
        int cr = 0, step0 = 0;                                        // step0: steps of this CTA before the item
        for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
            const Item t = item_at<T>(u, i);
            const int c = t.c0 + (warp & 3) * 32 + lane, h0 = 2 * first_parent(u, t), h1 = 2 * end_parent(u, t);
            for (int y = t.y0; y < t.y1; ++y, ++cr) {
                const int s = cr % G::SLOTS;
                if (!mbar_wait_warp(dfull + 8 * s, (cr / G::SLOTS) & 1)) { ok = false; break; }
                tc_fence_after();
                const unsigned at = tmem + quarter + s * G::CELLS;
                unsigned v[G::CELLS];
#pragma unroll
                for (int q = 0; q < G::CELLS; q += 16) tc_ld16(at + q, *reinterpret_cast<unsigned (*)[16]>(&v[q]));
                if constexpr (G::F32) {
                    unsigned odd_rows[16], small[16];
                    tc_ld16(at + G::DSUM, odd_rows);
                    tc_ld16(at + 2 * G::DSUM, small);
                    tc_wait_ld();
                    tc_st16(at + G::DSUM, zeros);
                    tc_st16(at + 2 * G::DSUM, zeros);
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        v[q] = __float_as_uint((__uint_as_float(v[q]) + __uint_as_float(odd_rows[q])) + __uint_as_float(small[q]));
                } else {
                    tc_wait_ld();
                }
#pragma unroll
                for (int q = 0; q < G::CELLS; q += 16) tc_st16(at + q, zeros);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive(dempty + 8 * s);
                T *o = static_cast<T *>(a.out) + (((size_t)t.n * a.C + c) * a.Hout + y) * a.W + t.x0;
                float zero[4] = {0.f, 0.f, 0.f, 0.f};                 // stays zero while all sums are finite
#pragma unroll
                for (int q = 0; q < G::CELLS; ++q) zero[q & 3] = fmaf(__uint_as_float(v[q]), 0.f, zero[q & 3]);
                if (!((zero[0] + zero[1]) + (zero[2] + zero[3]) == 0.f) && c < a.C) noted.note_sum(warp & 3, step0 + min(max(2 * (y - a.top), h0), h1 - 1) - h0);
                constexpr int PER = 16 / (int)sizeof(T);
#pragma unroll
                for (int q = 0; q < G::CELLS; q += PER)
                    if (c < a.C && t.x0 + q < a.W) {
                        uint4 w;
                        if constexpr (G::F32) {
                            w = make_uint4(v[q], v[q + 1], v[q + 2], v[q + 3]);
                        } else {
                            w.x = pack_pair(T(), __uint_as_float(v[q]), __uint_as_float(v[q + 1]));
                            w.y = pack_pair(T(), __uint_as_float(v[q + 2]), __uint_as_float(v[q + 3]));
                            w.z = pack_pair(T(), __uint_as_float(v[q + 4]), __uint_as_float(v[q + 5]));
                            w.w = pack_pair(T(), __uint_as_float(v[q + 6]), __uint_as_float(v[q + 7]));
                        }
                        *reinterpret_cast<uint4 *>(o + q) = w;
                    }
                __syncwarp();
            }
            step0 += h1 - h0;
        }
    }
    if (!ok) atomicExch(&g_wait_timeout, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == MMA_WARP) tc_dealloc(tmem, TMEM_COLS);
    if (warp < 8 && noted.last[warp & 3] >= 0) {                      // rare: outputs with something not finite (all are stored)
        int step0 = 0;
        for (int i = blockIdx.x; i < items; i += gridDim.x) {
            const Item t = item_at<T>(u, i);
            const int c = t.c0 + (warp & 3) * 32 + lane, h0 = 2 * first_parent(u, t), h1 = 2 * end_parent(u, t);
            for (int y = t.y0; y < t.y1; ++y) {
                // the high-res rows that reach this one and may be noted
                const int ha = max(2 * (y - a.top - 2), h0), hb = min(2 * (y - a.top + 3), h1);
                const int first = noted.first[warp & 3] - step0 + h0, last = noted.last[warp & 3] - step0 + h0;
                if ((y & 1) == warp >> 2 && c < a.C && hb > first && ha <= last)
                    finish_cells<T>(u, t.n, c, y, t.x0, max(ha, first), min(hb, last + 1), noted.sums[warp & 3] != 0);
            }
            step0 += h1 - h0;
        }
    }
}

}  // namespace gumma
