// sapa_proj_mm.cu — the projection (GroupNorm + 1x1 convolution, reference: sapa_base.py:27-34, sapa_deform.py:35-42) where the
// tcgen05 GEMM of sapa_proj.cu does not serve: in training, forward and backward, and for rows of any length and any d.
//
// Forward, two launches: proj_stats_kernel (sums of x and x^2 by slices of the groups) and proj_fwd_kernel, whose loader
// normalises x on its way into shared memory.  Backward, three launches:
//   proj_moments_kernel  dW and sum_p dq by slices of the pixels; behind a norm it also forms dy = W^T dq of its tile and sums
//                        S1 = sum_p dy and S2 = sum_p dy x per channel - all that GroupNorm's backward needs of the tensor;
//   proj_fold_kernel     parameter gradients (slices added in a fixed order, no atomics) and the coefficients
//                        alpha = -rstd^2 m2, delta = rstd (rstd mean m2 - m1) of
//   proj_dx_kernel       dx = rstd gamma_c dy + alpha_g x + delta_g (+ one more gradient of x), dy formed again from dq.
// The normalised tensor, its gradient and the casts between them never exist in memory (torch: about forty launches for the two
// projections of a module).  The projections of a module share the launches: a launch takes a list of problems.
//
// Rounding is that of the torch sequence these replace: with a 16-bit output type the normalised input, the weights, the product
// before the bias and dy are rounded to it (16-bit operands are exact in tf32, sums are float32); in float32 all products are
// three-term tf32 (1e-6).
#include "tma_util.cuh"

#include <algorithm>
#include <type_traits>

#include "proj_mm.h"

namespace sapa {
namespace pmm {

using namespace tmau;

constexpr int THREADS = 256;

// IN_ORDER: the kernel starts when the previous one has ended, so what it reads does not change while it runs (see begin_after_previous)
template <bool IN_ORDER, typename T> __device__ __forceinline__ T fetch_once(const T *p) {
    if constexpr (IN_ORDER) return __ldg(p);
    else return *p;
}
// 8 consecutive elements of a row, the ones from `valid` on as zeros
template <bool IN_ORDER = false, typename T> __device__ __forceinline__ void load8(const T *p, int valid, bool vec, float (&v)[8]) {
    if (vec && valid >= 8) {
        if constexpr (sizeof(T) == 4) {
            const float4 a = fetch_once<IN_ORDER>(reinterpret_cast<const float4 *>(p)), b = fetch_once<IN_ORDER>(reinterpret_cast<const float4 *>(p) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            const uint4 u = fetch_once<IN_ORDER>(reinterpret_cast<const uint4 *>(p));
            const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if constexpr (std::is_same<T, __half>::value) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
                    v[2 * i] = f.x; v[2 * i + 1] = f.y;
                } else {
                    v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
                }
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = i < valid ? to_acc(fetch_once<IN_ORDER>(p + i)) : 0.f;
    }
}
__device__ __forceinline__ void sts8(unsigned addr, const float (&v)[8]) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr + 16), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// v rounded to the type R and widened again
template <typename R> __device__ __forceinline__ float rounded(float v) {
    if constexpr (sizeof(R) == 4) return v;
    else return to_acc(from_acc<R>(v));
}
// which problem of the list a block belongs to: blocks are numbered through, problem after problem
template <typename L> __device__ __forceinline__ int find_problem(const L &l, int &block) {
    int i = 0;
    while (i + 1 < l.count && block >= l.p[i].blocks) { block -= l.p[i].blocks; ++i; }
    return i;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------------- statistics
template <typename T>
__global__ void __launch_bounds__(THREADS) proj_stats_kernel(const __grid_constant__ StatList list) {
    begin_after_previous();
    __shared__ double sc[2][THREADS / 32];
    int block = blockIdx.x;
    const StatProblem &q = list.p[find_problem(list, block)];
    const int split = block % q.nsplit, bg = block / q.nsplit, tid = threadIdx.x;
    const T *base = static_cast<const T *>(q.x) + (size_t)bg * q.n;
    const long long octs = (q.n + 7) / 8, per = (octs + q.nsplit - 1) / q.nsplit, o0 = split * per, o1 = min(octs, o0 + per);
    double s = 0, ss = 0;
    for (long long o = o0 + tid; o < o1; o += 2 * THREADS) {
        float v[2][8];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const long long at = o + u * THREADS;
            load8(base + at * 8, at < o1 ? (int)min((long long)8, q.n - at * 8) : 0, q.vec, v[u]);
        }
        float fs = 0.f, fss = 0.f;
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int i = 0; i < 8; ++i) { fs += v[u][i]; fss += v[u][i] * v[u][i]; }
        s += fs; ss += fss;
    }
    s = warp_sum(s); ss = warp_sum(ss);
    if ((tid & 31) == 0) { sc[0][tid >> 5] = s; sc[1][tid >> 5] = ss; }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < THREADS / 32; ++w) { s += sc[0][w]; ss += sc[1][w]; }
        q.partial[(size_t)bg * q.nsplit + split] = make_double2(s, ss);
    }
}

// ---------------------------------------------------------------------------------- forward
// Block = (problem, image, MT rows of W, 128 pixels); K in chunks of 32: W rows with a pitch of 36 words, x rows (pixels
// contiguous) with a pitch of 136 words, both free of conflicts for the fragment loads; the next chunk waits in registers.
constexpr int MM_P = 128, MM_K = 32, MM_APITCH = 36, MM_XPITCH = 136;

template <typename T, typename TO, int MT>
__global__ void __launch_bounds__(THREADS, 3) proj_fwd_kernel(const __grid_constant__ FwdList list) {
    begin_after_previous();
    constexpr bool LO = sizeof(TO) == 4;                        // float32 output: three-term products
    constexpr int WM = MT / 32, NT = 16 / (8 / WM), WPX = 8 * NT;      // warps along the rows; 8-pixel tiles / pixels of a warp
    __shared__ __align__(16) float as[MT * MM_APITCH], xs[MM_K * MM_XPITCH];
    __shared__ float2 s_st[MAX_GROUPS];
    int block = blockIdx.x;
    const FwdProblem &m = list.p[find_problem(list, block)];
    const int pb = block % m.pblocks; block /= m.pblocks;
    const int mb = block % m.mblocks, b = block / m.mblocks;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int HW = m.HW, p0 = pb * MM_P, m0 = mb * MT;
    const unsigned as_addr = (unsigned)__cvta_generic_to_shared(as), xs_addr = (unsigned)__cvta_generic_to_shared(xs);
    const int xrow = tid >> 4, xcol = (tid & 15) * 8;          // x: rows xrow, xrow + 16, pixels xcol .. xcol + 7
    const int arow = tid >> 3, acol = (tid & 7) * 4;           // W: rows arow (, arow + 32), columns acol .. acol + 3
    const T *W = static_cast<const T *>(m.weight);
    float xv[2][8], av[WM][4];
    const auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = k0 + xrow + 16 * i;
            load8(static_cast<const T *>(m.x) + ((size_t)b * m.K + k) * HW + p0 + xcol, k < m.K ? HW - p0 - xcol : 0, m.vec_x, xv[i]);
        }
#pragma unroll
        for (int i = 0; i < WM; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = m0 + arow + 32 * i, k = k0 + acol + e;
                av[i][e] = r < m.M && k < m.K ? rounded<TO>(to_acc(W[(size_t)r * m.K + k])) : 0.f;
            }
    };
    fetch(0);
    if (m.partial != nullptr)
        for (int i = tid; i < m.groups; i += THREADS) {
            double s = 0, ss = 0;
            for (int j = 0; j < m.nsplit; ++j) {
                const double2 v = m.partial[((size_t)b * m.groups + i) * m.nsplit + j];
                s += v.x; ss += v.y;
            }
            const double mean = s / (double)m.n, var = fmax(ss / (double)m.n - mean * mean, 0.0);
            s_st[i] = make_float2((float)mean, (float)(1.0 / sqrt(var + (double)m.eps)));
            if (m.stats != nullptr && pb == 0 && mb == 0) m.stats[(size_t)b * m.groups + i] = s_st[i];
        }
    float acc[2][NT][4] = {};
    const int wm = warp % WM, wp = warp / WM;
    for (int k0 = 0; k0 < m.K; k0 += MM_K) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = k0 + xrow + 16 * i;
            if (m.partial != nullptr && k < m.K) {
                const float2 st = s_st[k / m.cpg];
                const float a = st.y * to_acc(static_cast<const T *>(m.gamma)[k]), s = fmaf(-a, st.x, to_acc(static_cast<const T *>(m.beta)[k]));
#pragma unroll
                for (int e = 0; e < 8; ++e) xv[i][e] = fmaf(a, xv[i][e], s);
            }
            if (!LO)
#pragma unroll
                for (int e = 0; e < 8; ++e) xv[i][e] = rounded<TO>(xv[i][e]);
            sts8(xs_addr + 4 * ((xrow + 16 * i) * MM_XPITCH + xcol), xv[i]);
        }
#pragma unroll
        for (int i = 0; i < WM; ++i)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(as_addr + 4 * ((arow + 32 * i) * MM_APITCH + acol)), "f"(av[i][0]), "f"(av[i][1]),
                         "f"(av[i][2]), "f"(av[i][3]) : "memory");
        __syncthreads();
        if (k0 + MM_K < m.K) fetch(k0 + MM_K);
#pragma unroll
        for (int k = 0; k < MM_K; k += 8) {
            unsigned a[2][4], al[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float *p = as + (32 * wm + 16 * i + g) * MM_APITCH + k + t;
                a[i][0] = __float_as_uint(p[0]); a[i][1] = __float_as_uint(p[8 * MM_APITCH]);
                a[i][2] = __float_as_uint(p[4]); a[i][3] = __float_as_uint(p[8 * MM_APITCH + 4]);
                if (LO)
#pragma unroll
                    for (int e = 0; e < 4; ++e) al[i][e] = tf32_lo(a[i][e]);
            }
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float *p = xs + (k + t) * MM_XPITCH + WPX * wp + 8 * n + g;
                const unsigned b0 = __float_as_uint(p[0]), b1 = __float_as_uint(p[4 * MM_XPITCH]);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    mma_tf32(acc[i][n], a[i], b0, b1);
                    if (LO) {
                        mma_tf32(acc[i][n], al[i], b0, b1);
                        mma_tf32(acc[i][n], a[i], tf32_lo(b0), tf32_lo(b1));
                    }
                }
            }
        }
    }
    // D fragment: d0, d1 = (row g, pixels 2t, 2t + 1), d2, d3 = row g + 8
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = m0 + 32 * wm + 16 * i + 8 * half + g;
            if (r >= m.M) continue;
            const float bias = m.bias != nullptr ? rounded<TO>(to_acc(static_cast<const T *>(m.bias)[r])) : 0.f;
            TO *row = static_cast<TO *>(m.out) + ((size_t)b * m.M + r) * HW;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int p = p0 + WPX * wp + 8 * n + 2 * t;
                const float o0 = rounded<TO>(acc[i][n][2 * half]) + bias, o1 = rounded<TO>(acc[i][n][2 * half + 1]) + bias;
                if (m.pair && p + 1 < HW) store_pair<TO>(row + p, o0, o1);
                else {
                    if (p < HW) row[p] = from_acc<TO>(o0);
                    if (p + 1 < HW) row[p + 1] = from_acc<TO>(o1);
                }
            }
        }
}

// ---------------------------------------------------------------------------------- backward: moments
// Block = (problem, image, 64 channels, 64 rows of dq, slice of the pixels): dW[64 j x 64 c] += dq[64 j x 64 p] norm(x)[64 c x 64 p]^T,
// and with NORM (all rows of dq in one block) dy[64 c x 64 p] = W^T[64 c x d] dq for the two sums.  Both tiles lie in shared
// memory as float32 rows of 64 pixels with a pitch of 68 words; x stays as it came and is normalised in the fragments (a lane
// holds two channels); the next tile is in registers while the tensor cores work on this one.
constexpr int MO_C = 64, MO_J = 64, MO_P = 64, MO_PITCH = 68;

template <typename T, typename TG, bool NORM>
__global__ void __launch_bounds__(THREADS, 2) proj_moments_kernel(const __grid_constant__ MomentList list) {
    begin_after_previous();
    constexpr bool LO = sizeof(TG) == 4;
    extern __shared__ __align__(16) float mo_smem[];
    float *xs = mo_smem, *gs = xs + MO_C * MO_PITCH, *ws = gs + MO_J * MO_PITCH;      // ws (NORM only) = W^T: row = channel, column = row of dq
    int block = blockIdx.x;
    const MomentProblem &m = list.p[find_problem(list, block)];
    const int split = block % m.nsplit; block /= m.nsplit;
    const int cb = block % m.cblocks; block /= m.cblocks;
    const int jb = block % m.jblocks, b = block / m.jblocks;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int row0 = tid >> 3, col = (tid & 7) * 8;            // this thread's part of a tile: rows row0, row0 + 32, pixels col .. col + 7
    const int HW = m.HW, p_end = min(HW, (split + 1) * m.slice);
    const unsigned xs_addr = (unsigned)__cvta_generic_to_shared(xs), gs_addr = (unsigned)__cvta_generic_to_shared(gs);
    const T *x[2];
    const TG *gr[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int c = cb * MO_C + row0 + 32 * i, j = jb * MO_J + row0 + 32 * i;
        x[i] = c < m.C ? static_cast<const T *>(m.x) + ((size_t)b * m.C + c) * HW : nullptr;
        gr[i] = j < m.d1 ? static_cast<const TG *>(m.g1) + ((size_t)b * m.d1 + j) * HW
                : j < m.d ? static_cast<const TG *>(m.g2) + ((size_t)b * (m.d - m.d1) + j - m.d1) * HW : nullptr;
    }
    float xv[2][8], gv[2][8];
    const auto fetch = [&](int p0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            load8<LO>(x[i] + p0 + col, x[i] != nullptr ? p_end - p0 - col : 0, m.vec_x, xv[i]);
            load8<LO>(gr[i] + p0 + col, gr[i] != nullptr ? p_end - p0 - col : 0, m.vec_g, gv[i]);
        }
    };
    fetch(split * m.slice);
    const int wm = warp & 3, wn = warp >> 2;                    // warp: 16 channels; 32 rows of dq, then 32 pixels of dy
    // normalisation of this lane's two channels: y = ya x + ys
    float ya[2] = {1.f, 1.f}, ys[2] = {0.f, 0.f};
    if (NORM) {
        for (int i = tid; i < MO_C * ((m.d + 7) & ~7); i += THREADS) {
            const int c = i & (MO_C - 1), j = i / MO_C, cc = cb * MO_C + c;
            const T *w = j < m.d1 ? static_cast<const T *>(m.w1) + (size_t)j * m.C : static_cast<const T *>(m.w2) + (size_t)(j - m.d1) * m.C;
            ws[c * MO_PITCH + j] = cc < m.C && j < m.d ? rounded<TG>(to_acc(fetch_once<LO>(w + cc))) : 0.f;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = min(m.C - 1, cb * MO_C + 16 * wm + g + 8 * h);
            const float2 st = m.stats[(size_t)b * m.groups + c / m.cpg];
            ya[h] = st.y * to_acc(static_cast<const T *>(m.gamma)[c]);
            ys[h] = fmaf(-ya[h], st.x, to_acc(static_cast<const T *>(m.beta)[c]));
        }
    }
    const auto operand = [&](float v, int h) -> unsigned {      // x of channel half h as it entered the product (beyond the slice dq is zero)
        return __float_as_uint(rounded<TG>(NORM ? fmaf(ya[h], v, ys[h]) : v));
    };
    float acc[4][4] = {}, rsum[2] = {}, s1[2] = {}, s2[2] = {};
    for (int p0 = split * m.slice; p0 < p_end; p0 += MO_P) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            sts8(xs_addr + 4 * ((row0 + 32 * i) * MO_PITCH + col), xv[i]);
            sts8(gs_addr + 4 * ((row0 + 32 * i) * MO_PITCH + col), gv[i]);
            rsum[i] += ((gv[i][0] + gv[i][1]) + (gv[i][2] + gv[i][3])) + ((gv[i][4] + gv[i][5]) + (gv[i][6] + gv[i][7]));
        }
        __syncthreads();
        if (p0 + MO_P < p_end) fetch(p0 + MO_P);
        const float *xa = xs + (16 * wm + g) * MO_PITCH + t, *gb = gs + (32 * wn + g) * MO_PITCH + t;
#pragma unroll
        for (int k = 0; k < MO_P; k += 8) {
            unsigned a[4], al[4];
            a[0] = operand(xa[k], 0); a[1] = operand(xa[8 * MO_PITCH + k], 1);
            a[2] = operand(xa[k + 4], 0); a[3] = operand(xa[8 * MO_PITCH + k + 4], 1);
            if (LO)
#pragma unroll
                for (int i = 0; i < 4; ++i) al[i] = tf32_lo(a[i]);
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const unsigned b0 = __float_as_uint(gb[8 * n * MO_PITCH + k]), b1 = __float_as_uint(gb[8 * n * MO_PITCH + k + 4]);
                mma_tf32(acc[n], a, b0, b1);
                if (LO) {
                    mma_tf32(acc[n], al, b0, b1);
                    mma_tf32(acc[n], a, tf32_lo(b0), tf32_lo(b1));
                }
            }
        }
        if constexpr (NORM) {
            float dy[4][4] = {};
            const float *wa = ws + (16 * wm + g) * MO_PITCH + t, *gp = gs + t * MO_PITCH + 32 * wn + g;
            for (int k = 0; k < m.d; k += 8) {
                unsigned a[4], al[4];
                a[0] = __float_as_uint(wa[k]); a[1] = __float_as_uint(wa[8 * MO_PITCH + k]);
                a[2] = __float_as_uint(wa[k + 4]); a[3] = __float_as_uint(wa[8 * MO_PITCH + k + 4]);
                if (LO)
#pragma unroll
                    for (int i = 0; i < 4; ++i) al[i] = tf32_lo(a[i]);
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const unsigned b0 = __float_as_uint(gp[k * MO_PITCH + 8 * n]), b1 = __float_as_uint(gp[(k + 4) * MO_PITCH + 8 * n]);
                    mma_tf32(dy[n], a, b0, b1);
                    if (LO) {
                        mma_tf32(dy[n], al, b0, b1);
                        mma_tf32(dy[n], a, tf32_lo(b0), tf32_lo(b1));
                    }
                }
            }
            const float *xr = xs + (16 * wm + g) * MO_PITCH + 32 * wn + 2 * t;      // dq is zero beyond the slice, hence dy too
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float v = rounded<TG>(dy[n][e]);
                    s1[e >> 1] += v;
                    s2[e >> 1] = fmaf(v, xr[(e >> 1) * 8 * MO_PITCH + 8 * n + (e & 1)], s2[e >> 1]);
                }
        }
    }
    // D fragment: d0, d1 = (channel g, rows 2t, 2t + 1 of dq), d2, d3 = channel g + 8
    const size_t part = (size_t)b * m.nsplit + split;
    float *dw = m.dw + part * m.d * m.C;
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = cb * MO_C + 16 * wm + g + 8 * (e >> 1), j = jb * MO_J + 32 * wn + 8 * n + 2 * t + (e & 1);
            if (c < m.C && j < m.d) dw[(size_t)j * m.C + c] = acc[n][e];
        }
    if (cb == 0)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float s = rsum[i];
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const int j = jb * MO_J + row0 + 32 * i;
            if ((tid & 7) == 0 && j < m.d) m.rsums[part * m.d + j] = s;
        }
    if constexpr (NORM) {                                       // the quads, then the two warps of a channel block
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                s1[h] += __shfl_xor_sync(0xffffffffu, s1[h], o);
                s2[h] += __shfl_xor_sync(0xffffffffu, s2[h], o);
            }
            if (t == 0) {
                xs[wn * MO_C + 16 * wm + g + 8 * h] = s1[h];
                gs[wn * MO_C + 16 * wm + g + 8 * h] = s2[h];
            }
        }
        __syncthreads();
        const int c = cb * MO_C + tid;
        if (tid < MO_C && c < m.C) m.sums[part * m.C + c] = make_float2(xs[tid] + xs[MO_C + tid], gs[tid] + gs[MO_C + tid]);
    }
}

// ---------------------------------------------------------------------------------- backward: the small sums
// Blocks of a problem: first the rows of W (256 channels each), then one per group of channels for gamma, beta and the tail.
template <typename T>
__global__ void __launch_bounds__(THREADS) proj_fold_kernel(const __grid_constant__ FoldList list) {
    begin_after_previous();
    __shared__ float sm[2][THREADS];
    int block = blockIdx.x;
    const FoldProblem &f = list.p[find_problem(list, block)];
    const int tid = threadIdx.x, slices = f.B * f.nsplit;
    if (block < f.wblocks) {
        const int cblocks = (f.C + THREADS - 1) / THREADS, j = block / cblocks, c = block % cblocks * THREADS + tid;
        if (c < f.C) {
            float s[4] = {};
            int i = 0;
            for (; i + 4 <= slices; i += 4)
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] += __ldcs(f.dw + ((size_t)(i + u) * f.d + j) * f.C + c);
            for (; i < slices; ++i) s[0] += f.dw[((size_t)i * f.d + j) * f.C + c];
            const float v = (s[0] + s[1]) + (s[2] + s[3]);
            if (j < f.d1) static_cast<T *>(f.grad_weight)[(size_t)j * f.C + c] = from_acc<T>(v);
            else static_cast<T *>(f.grad_weight2)[(size_t)(j - f.d1) * f.C + c] = from_acc<T>(v);
        }
        if (block % cblocks == 0 && tid < 32) {
            float s = 0.f;
            for (int i = tid; i < slices; i += 32) s += f.rsums[(size_t)i * f.d + j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (tid == 0) {
                if (j < f.d1) { if (f.grad_bias != nullptr) static_cast<T *>(f.grad_bias)[j] = from_acc<T>(s); }
                else if (f.grad_bias2 != nullptr) static_cast<T *>(f.grad_bias2)[j - f.d1] = from_acc<T>(s);
            }
        }
        return;
    }
    // group gi of every image: thread (channel of the group, image-strided), then fixed-order sums
    const int gi = block - f.wblocks, lanes = THREADS / f.cpg, cl = tid % f.cpg, il = tid / f.cpg, c = gi * f.cpg + cl;
    const float gamma = to_acc(static_cast<const T *>(f.gamma)[c]);
    float dgamma = 0.f, dbeta = 0.f;
    for (int b0 = 0; b0 < f.B; ++b0) {
        float u = 0.f, v = 0.f;
        if (il < lanes)
            for (int i = il; i < f.nsplit; i += lanes) {
                const float2 s = f.sums[((size_t)b0 * f.nsplit + i) * f.C + c];
                u += s.x; v += s.y;
            }
        sm[0][tid] = u; sm[1][tid] = v;
        __syncthreads();
        const float2 st = f.stats[(size_t)b0 * f.groups + gi];
        if (tid < f.cpg) {
            for (int i = 1; i < lanes; ++i) { u += sm[0][i * f.cpg + tid]; v += sm[1][i * f.cpg + tid]; }
            v = st.y * (v - st.x * u);                          // sum of dy times the normalised x
            dbeta += u; dgamma += v;
            sm[0][tid] = gamma * u; sm[1][tid] = gamma * v;     // columns of the first row: this thread's own
        }
        __syncthreads();
        if (tid == 0) {
            float m1 = 0.f, m2 = 0.f;
            for (int i = 0; i < f.cpg; ++i) { m1 += sm[0][i]; m2 += sm[1][i]; }
            const float n = (float)f.cpg * (float)f.HW;
            m1 /= n; m2 /= n;
            f.tail[(size_t)b0 * f.groups + gi] = make_float2(-st.y * st.y * m2, st.y * (st.y * st.x * m2 - m1));
        }
        __syncthreads();
    }
    if (tid < f.cpg) {
        static_cast<T *>(f.grad_gamma)[c] = from_acc<T>(dgamma);
        static_cast<T *>(f.grad_beta)[c] = from_acc<T>(dbeta);
    }
}

// ---------------------------------------------------------------------------------- backward: dx
// Block = (problem, image, 64 channels, 64 pixels), K = the rows of dq in chunks of 32; x and the added gradient are fetched
// before the products start.
constexpr int DX_M = 64, DX_P = 64, DX_XPITCH = 72;

template <typename T, typename TG>
__global__ void __launch_bounds__(THREADS, sizeof(TG) == 4 ? 2 : 3) proj_dx_kernel(const __grid_constant__ DxList list) {
    begin_after_previous();
    constexpr bool LO = sizeof(TG) == 4;
    __shared__ __align__(16) float as[DX_M * MM_APITCH], xs[MM_K * DX_XPITCH];
    int block = blockIdx.x;
    const DxProblem &m = list.p[find_problem(list, block)];
    const int pb = block % m.pblocks; block /= m.pblocks;
    const int mb = block % m.mblocks, b = block / m.mblocks;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int HW = m.HW, p0 = pb * DX_P, m0 = mb * DX_M;
    const unsigned xs_addr = (unsigned)__cvta_generic_to_shared(xs);
    const int xrow = tid >> 3, xcol = (tid & 7) * 8;
    const int ac = tid & 63, ak = tid >> 6;                    // W: channel ac, rows ak, ak + 4, ... of the chunk (coalesced along the channels)
    float xv[8], av[8];
    const auto fetch = [&](int k0) {
        const int kx = k0 + xrow;
        const TG *row = kx < m.d1 ? static_cast<const TG *>(m.g1) + ((size_t)b * m.d1 + kx) * HW
                                  : static_cast<const TG *>(m.g2) + ((size_t)b * (m.d - m.d1) + kx - m.d1) * HW;
        load8(row + p0 + xcol, kx < m.d ? HW - p0 - xcol : 0, m.vec_g, xv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = k0 + ak + 4 * i, c = m0 + ac;
            const T *w = k < m.d1 ? static_cast<const T *>(m.w1) + (size_t)k * m.C : static_cast<const T *>(m.w2) + (size_t)(k - m.d1) * m.C;
            av[i] = k < m.d && c < m.C ? rounded<TG>(to_acc(w[c])) : 0.f;
        }
    };
    fetch(0);
    const int wm = warp & 1, wp = warp >> 1;                    // warp: 32 channels, 16 pixels
    float2 xe[2][2][2], ad[2][2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = m0 + 32 * wm + 16 * i + 8 * h + g;
            const size_t row = ((size_t)b * m.C + c) * HW;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int p = p0 + 16 * wp + 8 * n + 2 * t;
                xe[i][h][n] = ad[i][h][n] = make_float2(0.f, 0.f);
                if (c >= m.C || p >= HW) continue;
                const T *xp = static_cast<const T *>(m.x) + row + p;
                const TG *ap = static_cast<const TG *>(m.add) + row + p;
                if (m.pair) {                                   // even rows on aligned bases: pairs
                    if (m.tail != nullptr) xe[i][h][n] = load_pair<T>(xp);
                    if (m.add != nullptr) ad[i][h][n] = load_pair<TG>(ap);
                } else {
                    if (m.tail != nullptr) { xe[i][h][n].x = to_acc(xp[0]); if (p + 1 < HW) xe[i][h][n].y = to_acc(xp[1]); }
                    if (m.add != nullptr) { ad[i][h][n].x = to_acc(ap[0]); if (p + 1 < HW) ad[i][h][n].y = to_acc(ap[1]); }
                }
            }
        }
    float scale[2][2], alpha[2][2], delta[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = m0 + 32 * wm + 16 * i + 8 * h + g;
            scale[i][h] = 1.f; alpha[i][h] = 0.f; delta[i][h] = 0.f;
            if (m.tail != nullptr && c < m.C) {
                const size_t at = (size_t)b * m.groups + c / m.cpg;
                const float2 tl = m.tail[at];
                scale[i][h] = m.stats[at].y * to_acc(static_cast<const T *>(m.gamma)[c]); alpha[i][h] = tl.x; delta[i][h] = tl.y;
            }
        }
    float acc[2][2][4] = {};
    for (int k0 = 0; k0 < m.d; k0 += MM_K) {
        __syncthreads();
        sts8(xs_addr + 4 * (xrow * DX_XPITCH + xcol), xv);
#pragma unroll
        for (int i = 0; i < 8; ++i) as[ac * MM_APITCH + ak + 4 * i] = av[i];
        __syncthreads();
        if (k0 + MM_K < m.d) fetch(k0 + MM_K);
#pragma unroll
        for (int k = 0; k < MM_K; k += 8) {
            unsigned a[2][4], al[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float *p = as + (32 * wm + 16 * i + g) * MM_APITCH + k + t;
                a[i][0] = __float_as_uint(p[0]); a[i][1] = __float_as_uint(p[8 * MM_APITCH]);
                a[i][2] = __float_as_uint(p[4]); a[i][3] = __float_as_uint(p[8 * MM_APITCH + 4]);
                if (LO)
#pragma unroll
                    for (int e = 0; e < 4; ++e) al[i][e] = tf32_lo(a[i][e]);
            }
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const float *p = xs + (k + t) * DX_XPITCH + 16 * wp + 8 * n + g;
                const unsigned b0 = __float_as_uint(p[0]), b1 = __float_as_uint(p[4 * DX_XPITCH]);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    mma_tf32(acc[i][n], a[i], b0, b1);
                    if (LO) {
                        mma_tf32(acc[i][n], al[i], b0, b1);
                        mma_tf32(acc[i][n], a[i], tf32_lo(b0), tf32_lo(b1));
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = m0 + 32 * wm + 16 * i + 8 * h + g;
            if (c >= m.C) continue;
            T *row = static_cast<T *>(m.out) + ((size_t)b * m.C + c) * HW;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int p = p0 + 16 * wp + 8 * n + 2 * t;
                if (p >= HW) continue;
                const float o0 = fmaf(scale[i][h], rounded<TG>(acc[i][n][2 * h]), fmaf(alpha[i][h], xe[i][h][n].x, delta[i][h])) + ad[i][h][n].x;
                const float o1 = fmaf(scale[i][h], rounded<TG>(acc[i][n][2 * h + 1]), fmaf(alpha[i][h], xe[i][h][n].y, delta[i][h])) + ad[i][h][n].y;
                if (m.pair) store_pair<T>(row + p, o0, o1);
                else {
                    row[p] = from_acc<T>(o0);
                    if (p + 1 < HW) row[p + 1] = from_acc<T>(o1);
                }
            }
        }
}

// ---------------------------------------------------------------------------------- host side
static size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }
static bool rows16(const void *p, long long row, int esize) { return p == nullptr || (aligned16(p) && (row * esize) % 16 == 0); }
static int stat_slices(int B, int groups) { return std::max(1, std::min(64, (148 * 8 + B * groups - 1) / (B * groups))); }

static size_t forward_bytes(const sapa_projection *q, int count) {
    size_t at = 0;
    for (int i = 0; i < count; ++i)
        if (q[i].groups > 0) at = round256(at + (size_t)q[i].B * q[i].groups * stat_slices(q[i].B, q[i].groups) * sizeof(double2));
    return std::max<size_t>(at, 256);
}

template <typename T, typename TO>
static int run_forward(const sapa_projection *q, int count, unsigned char *ws, cudaStream_t st) {
    StatList sl{};
    FwdList fl{};
    size_t at = 0;
    int sblocks = 0, fblocks = 0, rows = 0;
    for (int i = 0; i < count; ++i) rows = std::max(rows, q[i].d);
    const int mt = rows <= 32 ? 32 : 64;
    fl.count = count;
    for (int i = 0; i < count; ++i) {
        const sapa_projection &s = q[i];
        FwdProblem &f = fl.p[i];
        f.x = s.x; f.weight = s.weight; f.bias = s.bias; f.gamma = s.gamma; f.beta = s.beta; f.out = s.out; f.eps = s.eps;
        f.B = s.B; f.M = s.d; f.K = s.C; f.HW = s.HW; f.groups = std::max(s.groups, 1); f.cpg = s.C / f.groups;
        f.mblocks = ceil_div(s.d, mt); f.pblocks = ceil_div(s.HW, MM_P); f.blocks = s.B * f.mblocks * f.pblocks;
        f.vec_x = rows16(s.x, s.HW, sizeof(T));
        f.pair = s.HW % 2 == 0 && aligned16(s.out);
        fblocks += f.blocks;
        if (s.groups == 0) continue;
        StatProblem &t = sl.p[sl.count++];
        t.x = s.x; t.partial = reinterpret_cast<double2 *>(ws + at); t.n = (long long)f.cpg * s.HW; t.nsplit = stat_slices(s.B, s.groups);
        t.blocks = s.B * s.groups * t.nsplit;
        t.vec = rows16(s.x, t.n, sizeof(T));
        at = round256(at + (size_t)t.blocks * sizeof(double2));
        sblocks += t.blocks;
        f.partial = t.partial; f.nsplit = t.nsplit; f.n = t.n; f.stats = static_cast<float2 *>(s.stats);
    }
    if (sl.count > 0) {
        launch_next(proj_stats_kernel<T>, sblocks, THREADS, 0, st, sl);
        if (int e = check_launch("proj_stats_kernel")) return e;
    }
    // The float32 forms, three products an element, have long blocks, of which a grid of less than a wave set up ahead makes an uneven
    // load: 3 x 192 x 25x31, 64 rows: 23 us in order, 38 ahead.
    if (sizeof(TO) == 4) launch_in_order(mt == 32 ? proj_fwd_kernel<T, TO, 32> : proj_fwd_kernel<T, TO, 64>, fblocks, THREADS, 0, st, fl);
    else launch_next(mt == 32 ? proj_fwd_kernel<T, TO, 32> : proj_fwd_kernel<T, TO, 64>, fblocks, THREADS, 0, st, fl);
    return check_launch("proj_fwd_kernel");
}

// Pixel slices of the moments: as many tiles per block as leave two blocks for every SM over all problems (a block first loads
// its rows of W and ends with its sums: more and shorter blocks measured 47 instead of 39 us for two 256-channel projections).
static int moment_tiles(const sapa_projection_grad *q, int count) {
    long long tiles = 0;
    for (int i = 0; i < count; ++i) tiles += (long long)q[i].B * ceil_div(q[i].C, MO_C) * ceil_div(q[i].d + q[i].d2, MO_J) * ceil_div(q[i].HW, MO_P);
    return ceil_div(tiles, 2 * 148);
}
static void plan_moments(MomentProblem &m, int tiles_per_block) {
    m.cblocks = ceil_div(m.C, MO_C);
    m.jblocks = ceil_div(m.d, MO_J);
    m.slice = std::min(tiles_per_block, ceil_div(m.HW, MO_P)) * MO_P;
    m.nsplit = ceil_div(m.HW, m.slice);
    m.blocks = m.B * m.cblocks * m.jblocks * m.nsplit;
}

struct BwdLayout { size_t dw, rsums, sums, tail, total; };
static BwdLayout bwd_layout(const MomentProblem &m, size_t at) {
    BwdLayout l;
    const auto take = [&](size_t floats) { const size_t r = at; at = round256(at + floats * sizeof(float)); return r; };
    const size_t parts = (size_t)m.B * m.nsplit;
    l.dw = take(parts * m.d * m.C);
    l.rsums = take(parts * m.d);
    l.sums = take(parts * m.C * 2);
    l.tail = take((size_t)m.B * m.groups * 2);
    l.total = at;
    return l;
}
static MomentProblem moment_problem(const sapa_projection_grad &q, int tiles_per_block) {
    MomentProblem m{};
    m.B = q.B; m.C = q.C; m.d = q.d + q.d2; m.d1 = q.d; m.HW = q.HW;
    m.groups = std::max(q.groups, 1); m.cpg = q.C / m.groups;
    plan_moments(m, tiles_per_block);
    return m;
}
static bool bwd_supported(const sapa_projection_grad &q) {
    return q.B > 0 && q.C > 0 && q.HW > 0 && q.d > 0 && q.d2 >= 0 && q.groups >= 0 && q.groups <= MAX_GROUPS &&
           (q.groups == 0 || (q.C % q.groups == 0 && q.C / q.groups <= THREADS && q.d + q.d2 <= MAX_D_NORM));
}

template <typename T, typename TG>
static int run_backward(const sapa_projection_grad *q, int count, unsigned char *ws, cudaStream_t st) {
    MomentList ml[2] = {};             // without and with a norm: two kernels
    FoldList fl{};
    DxList dl{};
    size_t at = 0;
    int mblocks[2] = {}, fblocks = 0, dblocks = 0;
    fl.count = count;
    const int tiles = moment_tiles(q, count);
    for (int i = 0; i < count; ++i) {
        const sapa_projection_grad &s = q[i];
        const int norm = s.groups > 0 ? 1 : 0;
        MomentProblem m = moment_problem(s, tiles);
        const BwdLayout l = bwd_layout(m, at);
        at = l.total;
        m.x = s.x; m.g1 = s.grad_out; m.g2 = s.grad_out2; m.w1 = s.weight; m.w2 = s.weight2; m.gamma = s.gamma; m.beta = s.beta;
        m.stats = norm ? static_cast<const float2 *>(s.stats) : nullptr;
        m.dw = reinterpret_cast<float *>(ws + l.dw); m.rsums = reinterpret_cast<float *>(ws + l.rsums); m.sums = reinterpret_cast<float2 *>(ws + l.sums);
        m.vec_x = rows16(s.x, s.HW, sizeof(T));
        m.vec_g = rows16(s.grad_out, s.HW, sizeof(TG)) && rows16(s.grad_out2, s.HW, sizeof(TG));
        ml[norm].p[ml[norm].count++] = m;
        mblocks[norm] += m.blocks;
        FoldProblem &f = fl.p[i];
        f.dw = m.dw; f.rsums = m.rsums; f.sums = m.sums; f.stats = m.stats; f.gamma = s.gamma; f.tail = reinterpret_cast<float2 *>(ws + l.tail);
        f.grad_weight = s.grad_weight; f.grad_weight2 = s.grad_weight2; f.grad_bias = s.grad_bias; f.grad_bias2 = s.grad_bias2;
        f.grad_gamma = s.grad_gamma; f.grad_beta = s.grad_beta;
        f.B = s.B; f.C = s.C; f.d = m.d; f.d1 = s.d; f.HW = s.HW; f.nsplit = m.nsplit; f.groups = m.groups; f.cpg = m.cpg;
        f.wblocks = m.d * ceil_div(s.C, THREADS);
        f.blocks = f.wblocks + (norm ? s.groups : 0);
        fblocks += f.blocks;
        if (s.grad_x == nullptr) continue;
        DxProblem &d = dl.p[dl.count++];
        d.x = s.x; d.g1 = s.grad_out; d.g2 = s.grad_out2; d.w1 = s.weight; d.w2 = s.weight2; d.gamma = s.gamma; d.add = s.add;
        d.stats = m.stats; d.tail = norm ? f.tail : nullptr; d.out = s.grad_x;
        d.B = s.B; d.C = s.C; d.d = m.d; d.d1 = s.d; d.HW = s.HW; d.groups = m.groups; d.cpg = m.cpg;
        d.mblocks = ceil_div(s.C, DX_M); d.pblocks = ceil_div(s.HW, DX_P); d.blocks = s.B * d.mblocks * d.pblocks;
        d.vec_g = m.vec_g;
        d.pair = s.HW % 2 == 0 && aligned16(s.x) && aligned16(s.grad_x) && (s.add == nullptr || aligned16(s.add));
        dblocks += d.blocks;
    }
    constexpr int smem_norm = 3 * MO_C * MO_PITCH * 4, smem_plain = 2 * MO_C * MO_PITCH * 4;
    int sms = 0;
    // float32 in order, as above, and then with __ldg: 16 x 128 x 64x64 with a norm 192 us, ahead 200, ahead with plain loads 228
    if (ml[1].count > 0) {
        if (int e = prepare_launch(reinterpret_cast<const void *>(proj_moments_kernel<T, TG, true>), smem_norm, "proj_moments_kernel", sms)) return e;
        if (sizeof(TG) == 4) launch_in_order(proj_moments_kernel<T, TG, true>, mblocks[1], THREADS, smem_norm, st, ml[1]);
        else launch_next(proj_moments_kernel<T, TG, true>, mblocks[1], THREADS, smem_norm, st, ml[1]);
        if (int e = check_launch("proj_moments_kernel")) return e;
    }
    if (ml[0].count > 0) {
        if (sizeof(TG) == 4) launch_in_order(proj_moments_kernel<T, TG, false>, mblocks[0], THREADS, smem_plain, st, ml[0]);
        else launch_next(proj_moments_kernel<T, TG, false>, mblocks[0], THREADS, smem_plain, st, ml[0]);
        if (int e = check_launch("proj_moments_kernel")) return e;
    }
    launch_next(proj_fold_kernel<T>, fblocks, THREADS, 0, st, fl);
    if (int e = check_launch("proj_fold_kernel")) return e;
    if (dl.count == 0) return SAPA_OK;
    launch_next(proj_dx_kernel<T, TG>, dblocks, THREADS, 0, st, dl);
    return check_launch("proj_dx_kernel");
}

}  // namespace pmm
}  // namespace sapa

using namespace sapa;

extern "C" {

size_t sapa_projections_workspace(const sapa_projection *p, int count) {
    if (p == nullptr || count < 1 || count > pmm::MAX_PROBLEMS) return 0;
    for (int i = 0; i < count; ++i)
        if (p[i].B <= 0 || p[i].C <= 0 || p[i].HW <= 0 || p[i].d <= 0 || p[i].groups < 0 || p[i].groups > pmm::MAX_GROUPS || (p[i].groups > 0 && p[i].C % p[i].groups != 0))
            return 0;
    return pmm::forward_bytes(p, count);
}

int sapa_projections_forward(const sapa_projection *p, int count, void *workspace, size_t workspace_bytes, int dtype, int out_dtype, void *stream) {
    const char *fn = "sapa_projections_forward";
    trace_reset();
    const size_t need = sapa_projections_workspace(p, count);
    SAPA_REQUIRE(need != 0, SAPA_ERR_UNSUPPORTED, "%s: needs 1 to %d problems of positive sizes, C divisible by groups, at most %d groups", fn,
                 pmm::MAX_PROBLEMS, pmm::MAX_GROUPS);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 256 == 0, SAPA_ERR_WORKSPACE,
                 "%s: a 256-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    for (int i = 0; i < count; ++i)
        SAPA_REQUIRE(p[i].x != nullptr && p[i].weight != nullptr && p[i].out != nullptr && (p[i].groups == 0 || (p[i].gamma != nullptr && p[i].beta != nullptr)),
                     SAPA_ERR_ARGUMENT, "%s: a pointer of problem %d is NULL", fn, i);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    if (dtype == SAPA_F32 && out_dtype == SAPA_F32) return pmm::run_forward<float, float>(p, count, ws, st);
    if (dtype == SAPA_F32 && out_dtype == SAPA_F16) return pmm::run_forward<float, __half>(p, count, ws, st);
    if (dtype == SAPA_F32 && out_dtype == SAPA_BF16) return pmm::run_forward<float, __nv_bfloat16>(p, count, ws, st);
    if (dtype == SAPA_F16 && out_dtype == SAPA_F16) return pmm::run_forward<__half, __half>(p, count, ws, st);
    if (dtype == SAPA_BF16 && out_dtype == SAPA_BF16) return pmm::run_forward<__nv_bfloat16, __nv_bfloat16>(p, count, ws, st);
    set_error("%s: no kernel for dtype codes %d / %d", fn, dtype, out_dtype);
    return SAPA_ERR_DTYPE;
}

size_t sapa_projections_backward_workspace(const sapa_projection_grad *p, int count) {
    if (p == nullptr || count < 1 || count > pmm::MAX_PROBLEMS) return 0;
    for (int i = 0; i < count; ++i)
        if (!pmm::bwd_supported(p[i])) return 0;
    size_t at = 0;
    const int tiles = pmm::moment_tiles(p, count);
    for (int i = 0; i < count; ++i) at = pmm::bwd_layout(pmm::moment_problem(p[i], tiles), at).total;
    return at;
}

int sapa_projections_backward(const sapa_projection_grad *p, int count, void *workspace, size_t workspace_bytes, int dtype, int grad_dtype,
                              void *stream) {
    const char *fn = "sapa_projections_backward";
    trace_reset();
    const size_t need = sapa_projections_backward_workspace(p, count);
    SAPA_REQUIRE(need != 0, SAPA_ERR_UNSUPPORTED, "%s: needs 1 to %d problems of positive sizes; behind a norm C divisible by groups, at most %d channels per "
                 "group and %d rows of W", fn, pmm::MAX_PROBLEMS, pmm::THREADS, pmm::MAX_D_NORM);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 256 == 0, SAPA_ERR_WORKSPACE,
                 "%s: a 256-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    for (int i = 0; i < count; ++i) {
        const sapa_projection_grad &s = p[i];
        SAPA_REQUIRE(s.x != nullptr && s.grad_out != nullptr && s.weight != nullptr && s.grad_weight != nullptr &&
                     (s.d2 == 0 || (s.grad_out2 != nullptr && s.weight2 != nullptr && s.grad_weight2 != nullptr)) &&
                     (s.groups == 0 || (s.gamma != nullptr && s.beta != nullptr && s.stats != nullptr && s.grad_gamma != nullptr && s.grad_beta != nullptr)),
                     SAPA_ERR_ARGUMENT, "%s: a pointer of problem %d is NULL", fn, i);
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    if (dtype == SAPA_F32 && grad_dtype == SAPA_F32) return pmm::run_backward<float, float>(p, count, ws, st);
    if (dtype == SAPA_F32 && grad_dtype == SAPA_F16) return pmm::run_backward<float, __half>(p, count, ws, st);
    if (dtype == SAPA_F32 && grad_dtype == SAPA_BF16) return pmm::run_backward<float, __nv_bfloat16>(p, count, ws, st);
    if (dtype == SAPA_F16 && grad_dtype == SAPA_F16) return pmm::run_backward<__half, __half>(p, count, ws, st);
    if (dtype == SAPA_BF16 && grad_dtype == SAPA_BF16) return pmm::run_backward<__nv_bfloat16, __nv_bfloat16>(p, count, ws, st);
    set_error("%s: no kernel for dtype codes %d / %d", fn, dtype, grad_dtype);
    return SAPA_ERR_DTYPE;
}

}  // extern "C"
