// sapa_d.cu — SAPA-D (deformable) kernels: similarity and aggregation at per-pixel learned sampling
// points, forward and backward, plus the fused forward.
//
// Every high-res pixel (qh, qw) samples, for each group g and point p, the low-res key / value plane at
//   (h, w) = (qh / s + off_h, qw / s + off_w)          off_w = offset[b, 2(gP+p)], off_h = offset[b, 2(gP+p)+1]
// bilinearly; a corner outside the plane reads 0 and a point outside (-1,H) x (-1,W) contributes nothing
// (forward and backward).  Because the sampling positions are data dependent the key/value gradients are a
// scatter: they use float atomics into a float32 (float64 for f64) accumulation buffer.  The gradients of
// the query, the attention and the offsets are owned by one thread each and written without atomics
// (query: P threads of a group add to one element, so it accumulates too).
#include "common.cuh"

#include <type_traits>

namespace sapa {

constexpr int MAXP = 16;   // largest num_point handled by the fused kernel

// Bilinear footprint of one sampling point in an H x W plane.  IN_ORDER: the kernel starts when the previous one has ended, so what it
// reads does not change while it runs (see begin_after_previous).
template <typename A, bool IN_ORDER = false>
struct Bilinear {
    int i00, i01, i10, i11;   // plane offsets of the four corners, -1 when the corner is outside
    A w00, w01, w10, w11;     // corner weights
    A lh, lw;                 // fractional parts (for the offset derivatives)
    bool inside;              // the reference's outer guard: -1 < h < H and -1 < w < W

    __device__ __forceinline__ void setup(A h, A w, int H, int W) {
        inside = (h > A(-1)) && (h < A(H)) && (w > A(-1)) && (w < A(W));
        const A fh = floor(h), fw = floor(w);
        const int h0 = (int)fh, w0 = (int)fw, h1 = h0 + 1, w1 = w0 + 1;
        lh = h - fh;
        lw = w - fw;
        const A hh = A(1) - lh, hw = A(1) - lw;
        w00 = hh * hw; w01 = hh * lw; w10 = lh * hw; w11 = lh * lw;
        const bool t = h0 >= 0, b = h1 <= H - 1, l = w0 >= 0, r = w1 <= W - 1;
        i00 = (inside && t && l) ? h0 * W + w0 : -1;
        i01 = (inside && t && r) ? h0 * W + w1 : -1;
        i10 = (inside && b && l) ? h1 * W + w0 : -1;
        i11 = (inside && b && r) ? h1 * W + w1 : -1;
    }
    template <typename T> static __device__ __forceinline__ T corner(const T *p) {
        if constexpr (IN_ORDER) return __ldg(p);
        else return *p;
    }
    template <typename T>
    __device__ __forceinline__ void corners(const T *plane, A &v00, A &v01, A &v10, A &v11) const {
        v00 = i00 >= 0 ? to_acc(corner(plane + i00)) : A(0);
        v01 = i01 >= 0 ? to_acc(corner(plane + i01)) : A(0);
        v10 = i10 >= 0 ? to_acc(corner(plane + i10)) : A(0);
        v11 = i11 >= 0 ? to_acc(corner(plane + i11)) : A(0);
    }
    template <typename T>
    __device__ __forceinline__ A sample(const T *plane) const {
        A v00, v01, v10, v11;
        corners(plane, v00, v01, v10, v11);
        return w00 * v00 + w01 * v01 + w10 * v10 + w11 * v11;
    }
};

// ---------------------------------------------------------------------------------- forward, separate ops

// one thread per (b, k = g*P+p, qh, qw)
template <typename T>
__global__ void deform_qk_fwd_kernel(const T *__restrict__ query, const T *__restrict__ key, const T *__restrict__ offset,
                                     T *__restrict__ out, int B, int Cq, int H, int W, int P, int s, int G) {
    using A = typename AccOf<T>::type;
    const int sH = s * H, sW = s * W, AC = G * P, gc = Cq / G;
    const size_t hi = (size_t)sH * sW, lo = (size_t)H * W;
    const long long total = (long long)B * AC * hi;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const size_t pix = (size_t)(i % hi);
        const int qw = (int)(pix % sW), qh = (int)(pix / sW);
        const int k = (int)((i / hi) % AC);
        const int b = (int)(i / (hi * AC));
        const int g = k / P;
        const T *op = offset + ((size_t)b * AC + k) * 2 * hi + pix;
        Bilinear<A, true> bl;
        bl.setup(A(qh / s) + to_acc(op[hi]), A(qw / s) + to_acc(op[0]), H, W);
        A acc = 0;
        if (bl.inside) {
            const T *qp = query + ((size_t)b * Cq + (size_t)g * gc) * hi + pix;
            const T *kp = key + ((size_t)b * Cq + (size_t)g * gc) * lo;
            for (int c = 0; c < gc; ++c) acc += bl.sample(kp + (size_t)c * lo) * to_acc(qp[(size_t)c * hi]);
        }
        out[i] = from_acc<T>(acc);
    }
}

// one thread per (b, chunk of CPT channels of one group, qh, qw): sampling set-up shared by CPT channels
template <typename T, int CPT>
__global__ void deform_av_fwd_kernel(const T *__restrict__ attn, const T *__restrict__ value, const T *__restrict__ offset,
                                     T *__restrict__ out, int B, int C, int H, int W, int P, int s, int G) {
    using A = typename AccOf<T>::type;
    const int sH = s * H, sW = s * W, AC = G * P, gc = C / G;
    const int chunks = (gc + CPT - 1) / CPT;
    const size_t hi = (size_t)sH * sW, lo = (size_t)H * W;
    const long long total = (long long)B * G * chunks * hi;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const size_t pix = (size_t)(i % hi);
        const int qw = (int)(pix % sW), qh = (int)(pix / sW);
        long long t = i / hi;
        const int ck = (int)(t % chunks); t /= chunks;
        const int g = (int)(t % G);
        const int b = (int)(t / G);
        const int c0 = g * gc + ck * CPT;
        const int nc = min(CPT, gc - ck * CPT);
        A o[CPT];
#pragma unroll
        for (int j = 0; j < CPT; ++j) o[j] = 0;
        const T *vp = value + ((size_t)b * C + c0) * lo;
        for (int p = 0; p < P; ++p) {
            const size_t k = (size_t)b * AC + (size_t)g * P + p;
            Bilinear<A, true> bl;
            bl.setup(A(qh / s) + to_acc(offset[k * 2 * hi + hi + pix]), A(qw / s) + to_acc(offset[k * 2 * hi + pix]), H, W);
            if (!bl.inside) continue;
            const A a = to_acc(attn[k * hi + pix]);
#pragma unroll
            for (int j = 0; j < CPT; ++j)
                if (j < nc) o[j] += bl.sample(vp + (size_t)j * lo) * a;
        }
#pragma unroll
        for (int j = 0; j < CPT; ++j)
            if (j < nc) out[((size_t)b * C + c0 + j) * hi + pix] = from_acc<T>(o[j]);
    }
}

// ---------------------------------------------------------------------------------- forward, fused
// A block of 32 x FY threads handles 32 consecutive pixels of one (image, group).  Phase 1: thread (x, y) computes
// the logits of points y, y + FY, ... of pixel x and leaves them, with the sampling positions, in shared memory.
// Phase 2: every thread normalises the P logits of its pixel (softmax over the points) and aggregates the value
// channels y*CPT .. of the group, CPT at a time.  The attention reaches HBM only if `attn_out` is given.
constexpr int FY = 8;

template <typename T, int CPT>
__global__ void __launch_bounds__(32 * FY)
deform_fused_fwd_kernel(const T *__restrict__ query, const T *__restrict__ key, const T *__restrict__ value,
                        const T *__restrict__ offset, T *__restrict__ out, T *__restrict__ attn_out,
                        int B, int Cq, int C, int H, int W, int P, int s, int G, int pix_blocks) {
    __shared__ float s_a[MAXP][32], s_h[MAXP][32], s_w[MAXP][32];
    const int sH = s * H, sW = s * W, AC = G * P, gq = Cq / G, gc = C / G;
    const size_t hi = (size_t)sH * sW, lo = (size_t)H * W;
    const int tx = threadIdx.x, ty = threadIdx.y;
    long long blk = blockIdx.x;
    const int pb = (int)(blk % pix_blocks); blk /= pix_blocks;
    const int g = (int)(blk % G);
    const int b = (int)(blk / G);
    const size_t pix = (size_t)pb * 32 + tx;
    const bool live = pix < hi;
    const int qw = live ? (int)(pix % sW) : 0, qh = live ? (int)(pix / sW) : 0;

    // phase 1: logits
    if (live) {
        const T *qp = query + ((size_t)b * Cq + (size_t)g * gq) * hi + pix;
        const T *kp = key + ((size_t)b * Cq + (size_t)g * gq) * lo;
        const T *op = offset + ((size_t)b * AC + (size_t)g * P) * 2 * hi + pix;
        for (int p = ty; p < P; p += FY) {
            const float w = float(qw / s) + to_acc(op[(size_t)(2 * p) * hi]);
            const float h = float(qh / s) + to_acc(op[(size_t)(2 * p + 1) * hi]);
            Bilinear<float, true> bl;
            bl.setup(h, w, H, W);
            float acc = 0.f;
            if (bl.inside)
                for (int c = 0; c < gq; ++c) acc += bl.sample(kp + (size_t)c * lo) * to_acc(qp[(size_t)c * hi]);
            s_a[p][tx] = acc;
            s_h[p][tx] = h;
            s_w[p][tx] = w;
        }
    }
    __syncthreads();
    if (!live) return;

    // phase 2: softmax over the points (every thread of the pixel's column does the same few operations)
    float m = -INFINITY;
    for (int p = 0; p < P; ++p) m = fmaxf(m, s_a[p][tx]);
    float z = 0.f;
    for (int p = 0; p < P; ++p) z += expf(s_a[p][tx] - m);
    const float inv = 1.f / z;
    if (attn_out != nullptr)
        for (int p = ty; p < P; p += FY)
            attn_out[((size_t)b * AC + (size_t)g * P + p) * hi + pix] = from_acc<T>(expf(s_a[p][tx] - m) * inv);

    for (int c0 = ty * CPT; c0 < gc; c0 += FY * CPT) {
        const T *vp = value + ((size_t)b * C + (size_t)g * gc + c0) * lo;
        const int nc = min(CPT, gc - c0);
        float o[CPT];
#pragma unroll
        for (int j = 0; j < CPT; ++j) o[j] = 0.f;
        for (int p = 0; p < P; ++p) {
            Bilinear<float, true> bl;
            bl.setup(s_h[p][tx], s_w[p][tx], H, W);
            if (!bl.inside) continue;
            const float a = expf(s_a[p][tx] - m) * inv;
#pragma unroll
            for (int j = 0; j < CPT; ++j)
                if (j < nc) o[j] += bl.sample(vp + (size_t)j * lo) * a;
        }
#pragma unroll
        for (int j = 0; j < CPT; ++j)
            if (j < nc) out[((size_t)b * C + (size_t)g * gc + c0 + j) * hi + pix] = from_acc<T>(o[j]);
    }
}

// ---------------------------------------------------------------------------------- backward
// one thread per (b, k, qh, qw), looping over the channels of group g(k).
//   QK: top = dS[b,k,pix], weight_c = Q[b,c,pix]:   dQ_c += top*val_c (atomic), dKey_c[corner] += w*top*Q_c (atomic)
//   AV: top_c = dOut[b,c,pix], weight = A[b,k,pix]: dA = sum_c top_c*val_c,     dV_c[corner]   += w*top_c*A (atomic)
// and in both: dOff_w = sum_c (d val_c / d w) * top * weight, dOff_h likewise.
template <typename T, bool IS_QK>
__global__ void deform_bwd_kernel(const T *__restrict__ top, const T *__restrict__ hires /* Q | A */,
                                  const T *__restrict__ plane_src /* Key | V */, const T *__restrict__ offset,
                                  typename AccOf<T>::type *__restrict__ grad_hi_acc /* dQ (QK only) */,
                                  T *__restrict__ grad_attn /* dA (AV only) */,
                                  typename AccOf<T>::type *__restrict__ grad_plane /* dKey | dV */,
                                  T *__restrict__ grad_offset, int B, int Cc, int H, int W, int P, int s, int G) {
    using A = typename AccOf<T>::type;
    const int sH = s * H, sW = s * W, AC = G * P, gc = Cc / G;
    const size_t hi = (size_t)sH * sW, lo = (size_t)H * W;
    const long long total = (long long)B * AC * hi;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const size_t pix = (size_t)(i % hi);
        const int qw = (int)(pix % sW), qh = (int)(pix / sW);
        const int k = (int)((i / hi) % AC);
        const int b = (int)(i / (hi * AC));
        const int g = k / P;
        const size_t off_idx = ((size_t)b * AC + k) * 2 * hi + pix;
        Bilinear<A, true> bl;
        bl.setup(A(qh / s) + to_acc(offset[off_idx + hi]), A(qw / s) + to_acc(offset[off_idx]), H, W);
        A g_w = 0, g_h = 0, g_attn = 0;
        if (bl.inside) {
            const A hh = A(1) - bl.lh, hw = A(1) - bl.lw;
            const size_t ch0 = (size_t)b * Cc + (size_t)g * gc;
            const A top_k = IS_QK ? to_acc(top[i]) : A(0);
            const A wt_k = IS_QK ? A(0) : to_acc(hires[i]);
            for (int c = 0; c < gc; ++c) {
                const T *pl = plane_src + (ch0 + c) * lo;
                A v00, v01, v10, v11;
                bl.corners(pl, v00, v01, v10, v11);
                const A val = bl.w00 * v00 + bl.w01 * v01 + bl.w10 * v10 + bl.w11 * v11;
                A t, wt;
                if (IS_QK) {
                    t = top_k;
                    wt = to_acc(hires[(ch0 + c) * hi + pix]);
                    atomic_add(grad_hi_acc + (ch0 + c) * hi + pix, t * val);
                } else {
                    t = to_acc(top[(ch0 + c) * hi + pix]);
                    wt = wt_k;
                    g_attn += t * val;
                }
                const A tw = t * wt;
                A *gp = grad_plane + (ch0 + c) * lo;
                if (bl.i00 >= 0) atomic_add(gp + bl.i00, bl.w00 * tw);
                if (bl.i01 >= 0) atomic_add(gp + bl.i01, bl.w01 * tw);
                if (bl.i10 >= 0) atomic_add(gp + bl.i10, bl.w10 * tw);
                if (bl.i11 >= 0) atomic_add(gp + bl.i11, bl.w11 * tw);
                g_w += (-hh * v00 + hh * v01 - bl.lh * v10 + bl.lh * v11) * tw;
                g_h += (-hw * v00 - bl.lw * v01 + hw * v10 + bl.lw * v11) * tw;
            }
        }
        grad_offset[off_idx] = from_acc<T>(g_w);
        grad_offset[off_idx + hi] = from_acc<T>(g_h);
        if (!IS_QK) grad_attn[i] = from_acc<T>(g_attn);
    }
}

// ---------------------------------------------------------------------------------- forward, dense-window path
// With s = 2 and offsets inside [-2, 2) a sampling point's four corners lie in the 5 x 5 low-res window around the
// pixel's parent - the window of SAPA-B.  Then both contractions of SAPA-D are SAPA-B contractions:
//   logits:      sim_p = sum_c q_c * bilinear(key_c) = sum_corners w_corner * D[corner],  D[cell] = sum_c q_c key_c[cell]
//                (D = the dense 25-slot similarity of the group's 16 channels, one call of the SAPA-B logit kernel with
//                the B x G groups as images);
//   aggregation: out_c = sum_p a_p * bilinear(value_c) = sum_cells Wd[cell] * value_c[cell],  Wd[cell] = sum of a_p * w_corner
//                over the corners that land on the cell (one call of the SAPA-B aggregation kernel).
// deform_window_kernel sits between the two: one thread per (image, group, pixel) turns D and the offsets into the
// attention over the P points and the dense window weights Wd (the thread's two windows sit in its column of a shared
// array, where the four cells of a point can be addressed at run time).  A point with a corner outside the window
// (|offset| >= 2) is an "outlier": its logit is gathered directly here, it adds nothing to Wd, and its pixel is
// appended to a list from which deform_outlier_kernel adds the contribution to the output afterwards (rare for learned
// offsets, but always correct).  Points outside the image contribute exactly 0 to the logits and to the output, as in
// the reference.
constexpr int WIN_THREADS = 128;

// One entry per (image, group, pixel) that has at least one point outside its window: the points as a bit mask and
// the attention weights of all points of the pixel.
struct OutlierTap {
    unsigned int idx;    // (image * G + group) * sH * sW + high-res pixel
    unsigned int mask;   // bit p: point p left the window
    float a[MAXP];       // attention weight of every point (only the masked ones are read)
};

// Position of a sampling point relative to the window of its pixel: r0 / c0 = window row / column of the upper-left
// corner, lh / lw the fractional parts; `dense` = all four corners are window cells, `inside` = the reference's guard.
struct WindowTap {
    int r0, c0;
    float lh, lw;
    bool inside, dense;
    __device__ __forceinline__ void setup(float h, float w, int H, int W, int py, int px) {
        inside = (h > -1.f) && (h < float(H)) && (w > -1.f) && (w < float(W));
        const float fh = floorf(h), fw = floorf(w);
        lh = h - fh; lw = w - fw;
        r0 = (int)fh - (py - 2); c0 = (int)fw - (px - 2);
        dense = inside && r0 >= 0 && r0 <= 3 && c0 >= 0 && c0 <= 3;
    }
};

// MODE: WIN_FUSED = logits -> softmax -> window weights (the fused op); WIN_WEIGHTS = window weights from a given attention map
// (deform_av).  Raw logits (deform_qk) have a kernel of their own.
constexpr int WIN_FUSED = 0, WIN_WEIGHTS = 1;

// The points of a pixel inside its window: fractional parts, and the place of the upper-left cell in the thread's column of a
// [25][WIN_THREADS] array, two points to a register.  Points that are not dense have place 0 and take no part (see `dense`); their
// fractional parts are 0 too: those of an infinite or undefined offset are NaN, which no weight of zero keeps out of a sum.
template <int PMAX>
struct WindowPoints {
    float lh[PMAX], lw[PMAX];
    unsigned place[(PMAX + 1) / 2], dense, outliers;
    __device__ __forceinline__ int at(int p) const { return (int)(p & 1 ? place[p >> 1] >> 16 : place[p >> 1] & 0xffffu); }
    float oh[PMAX], ow[PMAX];
    template <typename T>
    __device__ __forceinline__ void load(const T *offp, size_t hi, bool live, int P) {
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            const bool on = live && p < P;
            ow[p] = on ? to_acc(offp[(size_t)(2 * p) * hi]) : 0.f;
            oh[p] = on ? to_acc(offp[(size_t)(2 * p + 1) * hi]) : 0.f;
        }
        dense = outliers = 0u;
    }
    __device__ __forceinline__ void set(int p, bool on, int rows, int W, int py, int px) {
        WindowTap t;
        t.setup(float(py) + oh[p], float(px) + ow[p], rows, W, py, px);
        const bool in = on && t.dense;
        lh[p] = in ? t.lh : 0.f; lw[p] = in ? t.lw : 0.f;
        const unsigned c = in ? (unsigned)((t.r0 * 5 + t.c0) * WIN_THREADS) : 0u;
        place[p >> 1] = p & 1 ? place[p >> 1] | (c << 16) : c;
        dense |= in ? 1u << p : 0u;
        outliers |= on && t.inside && !t.dense ? 1u << p : 0u;
    }
};
template <int N> __device__ __forceinline__ void put(float (&v)[N], int p, float x) {      // at a place known at run time
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = j == p ? x : v[j];
}
// logit of a point outside the window: the key gathered directly
template <typename T>
__device__ __forceinline__ float far_logit(const T *query, const T *key, const T *offp, int p, size_t bg, int gq, size_t hi, size_t lo, size_t pix, int rows, int W,
                                           int py, int px) {
    Bilinear<float> bl;
    bl.setup(float(py) + to_acc(offp[(size_t)(2 * p + 1) * hi]), float(px) + to_acc(offp[(size_t)(2 * p) * hi]), rows, W);
    const T *qp = query + bg * gq * hi + pix, *kp = key + bg * gq * lo;
    float acc = 0.f;
    for (int ch = 0; ch < gq; ++ch) acc += bl.sample(kp + (size_t)ch * lo) * to_acc(qp[(size_t)ch * hi]);
    return acc;
}

// The two 25-slot windows of a thread (similarity in, window weights out) live in shared memory, column = thread, so
// every access is conflict-free: a point touches four cells of each window, and shared memory can be indexed with the
// cell computed at run time (a register array cannot: that form multiplies every point with all 25 cells and took
// 82 us at B=8, 4 groups, 128 x 128 pixels).  Two passes over the points: logits and their maximum, then exp and the window
// weights.  Bound by latency at 24 warps per SM (80 registers, of which the form for 9 points spills 20 and that for 16 points 60; 4 and
// 8 blocks measured slower), so the points go side by side: no branch on a point (what it must not add is selected away; outliers have a
// loop of their own), places kept from pass to pass, block = pixels of one (image, group) instead of 64-bit divisions per thread: 55 -> 43
// us (float32; bfloat16 59 -> 44).
//
// PMAX = the most points of an instance (see launch_window); 9 is the 3 x 3 points of the reference modules' default, exactly.
template <typename T, int PMAX, int MODE>
__global__ void __launch_bounds__(WIN_THREADS, 6)
deform_window_kernel(const T *query, const T *key, const T *offset,
                          const float *dense, T *attn, T *window,
                          OutlierTap *taps, unsigned int *tap_count, int B, int Cq, int H, int W,
                          int P_runtime, int G, int rows, int ytop) {
    begin_after_previous();
    __shared__ float sd[MODE == WIN_FUSED ? 25 : 1][WIN_THREADS];     // dense similarity of the thread's pixel
    __shared__ float sw[25][WIN_THREADS];                               // window weights being collected
    const int P = PMAX == 9 ? 9 : P_runtime;
    const unsigned sW = 2 * W;
    const int gq = Cq / G;
    const size_t hi = (size_t)(2 * H) * sW, lo = (size_t)rows * W;
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    const unsigned blocks = ((unsigned)hi + blockDim.x - 1) / blockDim.x, groups = (unsigned)(B * G);      // of an (image, group)
    float *const dcol = &sd[0][tid], *const wcol = &sw[0][tid];
    for (unsigned bg = blockIdx.y; bg < groups; bg += gridDim.y)
    for (unsigned block = blockIdx.x; block < blocks; block += gridDim.x) {
        const unsigned at_pix = block * blockDim.x + tid, pix = at_pix < hi ? at_pix : 0u;
        const bool live = at_pix < hi;
        const int qh = (int)(pix / sW), qw = (int)(pix - (unsigned)qh * sW), py = (qh >> 1) + ytop, px = qw >> 1;
        const T *offp = offset + (size_t)bg * P * 2 * hi + pix;
        if (MODE == WIN_FUSED) {
            const float *dp = dense + (size_t)bg * 25 * hi + pix;
#pragma unroll
            for (int k = 0; k < 25; ++k) dcol[k * WIN_THREADS] = live ? __ldcs(dp + (size_t)k * hi) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 25; ++k) wcol[k * WIN_THREADS] = 0.f;
        WindowPoints<PMAX> pts;
        pts.load(offp, hi, live, P);
        // ---- pass 1: logits (or the given attention)
        float logit[PMAX];
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            pts.set(p, live && p < P, rows, W, py, px);
            if (MODE == WIN_WEIGHTS) {
                logit[p] = live && p < P ? to_acc(attn[((size_t)bg * P + p) * hi + pix]) : 0.f;
            } else {
                const float *c = dcol + pts.at(p);
                const float top = (1.f - pts.lw[p]) * c[0] + pts.lw[p] * c[WIN_THREADS];
                const float bot = (1.f - pts.lw[p]) * c[5 * WIN_THREADS] + pts.lw[p] * c[6 * WIN_THREADS];
                logit[p] = pts.dense >> p & 1 ? (1.f - pts.lh[p]) * top + pts.lh[p] * bot : 0.f;
            }
        }
        if (MODE == WIN_FUSED)
            for (unsigned left = pts.outliers; left != 0; left &= left - 1) {      // outliers: gather the key directly
                const int p = __ffs(left) - 1;
                put(logit, p, far_logit(query, key, offp, p, bg, gq, hi, lo, pix, rows, W, py, px));
            }
        // ---- pass 2: exp and the window weights
        float m = -INFINITY, z = 0.f;
#pragma unroll
        for (int p = 0; p < PMAX; ++p)
            if (p < P) m = fmaxf(m, logit[p]);
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            const float e = p < P ? MODE == WIN_WEIGHTS ? logit[p] : __expf(logit[p] - m) : 0.f;
            logit[p] = e;
            z += e;
            const float add = pts.dense >> p & 1 ? e : 0.f, et = add * (1.f - pts.lh[p]), eb = add * pts.lh[p];
            float *c = wcol + pts.at(p);
            const float c00 = c[0], c01 = c[WIN_THREADS], c10 = c[5 * WIN_THREADS], c11 = c[6 * WIN_THREADS];
            c[0] = c00 + et * (1.f - pts.lw[p]);
            c[WIN_THREADS] = c01 + et * pts.lw[p];
            c[5 * WIN_THREADS] = c10 + eb * (1.f - pts.lw[p]);
            c[6 * WIN_THREADS] = c11 + eb * pts.lw[p];
        }
        const float inv = MODE == WIN_WEIGHTS ? 1.f : 1.f / z;
        if (live) {
            T *wp = window + (size_t)bg * 25 * hi + pix;
#pragma unroll
            for (int k = 0; k < 25; ++k) wp[(size_t)k * hi] = from_acc<T>(wcol[k * WIN_THREADS] * inv);
        }
        if (MODE == WIN_FUSED) {
#pragma unroll
            for (int p = 0; p < PMAX; ++p) {
                logit[p] *= inv;                             // the attention weight of the point
                if (live && p < P && attn != nullptr) attn[((size_t)bg * P + p) * hi + pix] = from_acc<T>(logit[p]);
            }
        }
        // append the pixels of this warp that have outlier points to the list: one counter update per warp
        const unsigned int any = __ballot_sync(0xffffffffu, pts.outliers != 0);
        if (any != 0) {
            unsigned int base = 0;
            if (lane == 0) base = atomicAdd(tap_count, (unsigned int)__popc(any));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (pts.outliers != 0) {
                OutlierTap *t = taps + base + __popc(any & ((1u << lane) - 1u));
                t->idx = (unsigned int)(bg * hi + pix);
                t->mask = pts.outliers;
#pragma unroll
                for (int p = 0; p < PMAX; ++p) t->a[p] = logit[p];
            }
        }
    }
}

// Raw logits of the separate op: one pass, nothing kept, each logit written as it is found.  Blocks run over the pixels of all (image,
// group)s in one row, and a point outside the window is gathered where it is met: with the blocks and the loop of far points of
// deform_window_kernel this pass is slower (float32, 8 x 4 groups x 128x128 pixels, with the similarity: 9 points 82 us, 64 this
// way; bfloat16 76 and 59).
template <typename T, int PMAX>
__global__ void __launch_bounds__(WIN_THREADS, 6)
deform_logits_kernel(const T *query, const T *key, const T *offset, const float *dense, T *out, int groups, int gq, int H, int W, int P_runtime) {
    begin_after_previous();
    __shared__ float sd[25][WIN_THREADS];                   // dense similarity of the thread's pixel
    const int P = PMAX == 9 ? 9 : P_runtime, tid = threadIdx.x;
    const size_t sW = 2 * (size_t)W, hi = 2 * (size_t)H * sW, lo = (size_t)H * W;
    const long long total = (long long)groups * hi;
    for (long long i0 = (long long)blockIdx.x * WIN_THREADS; i0 < total; i0 += (long long)gridDim.x * WIN_THREADS) {
        const long long i = i0 + tid;
        const bool live = i < total;
        const size_t pix = live ? (size_t)(i % hi) : 0;
        const long long bg = live ? i / (long long)hi : 0;
        const int py = (int)(pix / sW) >> 1, px = (int)(pix % sW) >> 1;
        const float *dp = dense + (size_t)bg * 25 * hi + pix;
#pragma unroll
        for (int k = 0; k < 25; ++k) sd[k][tid] = live ? __ldcs(dp + (size_t)k * hi) : 0.f;
        const T *offp = offset + (size_t)bg * P * 2 * hi + pix;
        float oh[PMAX], ow[PMAX];
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            const bool on = live && p < P;
            ow[p] = on ? float(px) + to_acc(offp[(size_t)(2 * p) * hi]) : 0.f;
            oh[p] = on ? float(py) + to_acc(offp[(size_t)(2 * p + 1) * hi]) : 0.f;
        }
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            if (live && p < P) {
                WindowTap t;
                t.setup(oh[p], ow[p], H, W, py, px);
                float v = 0.f;
                if (t.dense) {
                    const int c = t.r0 * 5 + t.c0;
                    const float top = (1.f - t.lw) * sd[c][tid] + t.lw * sd[c + 1][tid];
                    const float bot = (1.f - t.lw) * sd[c + 5][tid] + t.lw * sd[c + 6][tid];
                    v = (1.f - t.lh) * top + t.lh * bot;
                } else if (t.inside) {
                    v = far_logit(query, key, offp, p, (size_t)bg, gq, hi, lo, pix, H, W, py, px);
                }
                out[((size_t)bg * P + p) * hi + pix] = from_acc<T>(v);
            }
        }
    }
}

// Adds a_p * bilinear(value_c) of the listed outlier points to the output.  SUB threads per listed pixel: each takes
// every SUB-th channel of the group, CH channels at a time in registers, walks the pixel's outlier points for them
// and then updates the output elements once, read-modify-write without atomics (a listed pixel of a group belongs to
// exactly one thread group, and the aggregation kernel that wrote the output has finished): the forward pass is
// deterministic and a 16-bit output is rounded once more, not once per point.
template <int SUB, int CH, typename T>
__device__ __forceinline__ void outlier_pixels(const OutlierTap *taps, unsigned int n, const T *value,
                                               const T *offset, T *out, int C, int H, int W, int P, int G, int rows, int ytop) {
    const int sW = 2 * W, gc = C / G;
    const size_t hi = (size_t)(2 * H) * sW, lo = (size_t)rows * W;
    const int sub = threadIdx.x % SUB;
    // entries of a short list are spread over the blocks, those of a long one stay next to their neighbours
    const unsigned int first = SUB == 32 ? threadIdx.x / SUB * gridDim.x + blockIdx.x : (blockIdx.x * blockDim.x + threadIdx.x) / SUB;
    for (unsigned int e = first; e < n; e += gridDim.x * blockDim.x / SUB) {
        const OutlierTap *t = taps + e;
        const unsigned int idx = t->idx, mask = t->mask;
        const size_t bg = idx / hi, pix = idx % hi;
        const int px = (int)(pix % sW) >> 1, py = ((int)(pix / sW) >> 1) + ytop;
        const T *offp = offset + bg * P * 2 * hi + pix;
        const T *vp = value + bg * gc * lo;
        T *op = out + bg * gc * hi + pix;
        for (int c0 = sub; c0 < gc; c0 += SUB * CH) {
            float acc[CH], old[CH];
#pragma unroll
            for (int j = 0; j < CH; ++j) {
                acc[j] = 0.f;
                old[j] = c0 + SUB * j < gc ? to_acc(op[(size_t)(c0 + SUB * j) * hi]) : 0.f;
            }
            for (unsigned int m = mask; m != 0; m &= m - 1) {
                const int p = __ffs(m) - 1;
                const float w = float(px) + to_acc(offp[(size_t)(2 * p) * hi]);
                const float h = float(py) + to_acc(offp[(size_t)(2 * p + 1) * hi]);
                const float a = t->a[p];
                Bilinear<float> bl;
                bl.setup(h, w, rows, W);
#pragma unroll
                for (int j = 0; j < CH; ++j) {
                    const int c = c0 + SUB * j;
                    if (c < gc) acc[j] += a * bl.sample(vp + (size_t)c * lo);
                }
            }
#pragma unroll
            for (int j = 0; j < CH; ++j) {
                const int c = c0 + SUB * j;
                if (c < gc) op[(size_t)c * hi] = from_acc<T>(old[j] + acc[j]);
            }
        }
    }
}
// A short list (learned offsets: a few hundred entries) is a chain of dependent loads per entry: a warp per entry and every channel
// in flight at once (25 -> 7 us for 317 pixels of 64 channels in float16).  A long one is bound by its sectors, which neighbouring pixels
// share when eight threads serve each.
template <typename T>
__global__ void deform_outlier_kernel(const OutlierTap *taps, const unsigned int *tap_count,
                                      const T *value, const T *offset, T *out,
                                      int C, int H, int W, int P, int G, int rows, int ytop) {
    begin_after_previous();
    const unsigned int n = *tap_count;
    if (n <= gridDim.x * (blockDim.x / 32)) outlier_pixels<32, 2>(taps, n, value, offset, out, C, H, W, P, G, rows, ytop);
    else outlier_pixels<8, 4>(taps, n, value, offset, out, C, H, W, P, G, rows, ytop);
}

// ---------------------------------------------------------------------------------- backward, dense-window path
// The forward identities read backwards (B_p = the 25-vector of bilinear weights of point p, vy (x) vx):
//   dWd[cell]   = sum_c dOut_c * value_c[cell]              = sim(dOut, value) per group           (SAPA-B logit kernel)
//   dA_p        = sum_cells B_p[cell] * dWd[cell];   dS_p = A_p * (dA_p - sum_q A_q dA_q)           (softmax over the points)
//   dD[cell]    = sum_p dS_p * B_p[cell],  Wd[cell] = sum_p A_p * B_p[cell]
//   dQ = agg(dD, key),  dKey = gath(Q, dD),  dV = gath(dOut, Wd)  per group                         (SAPA-B kernels, no atomics)
//   d offset_p  = A_p * (dB_p . dWd) + dS_p * (dB_p . D),   dB_p/dh = dvy (x) vx,  dB_p/dw = vy (x) dvx
// deform_window_bwd_kernel does the per-pixel part (one thread per (image, group, pixel); the windows in shared memory).
// Points that leave the window are listed with their A_p and dS_p; deform_outlier_bwd_kernel adds their gradients
// afterwards (atomics on dQ, dKey, dV; it owns their offset gradients).
struct OutlierGrad {
    unsigned int k;      // (image * G + group) * P + point
    unsigned int pix;    // high-res pixel
    float a;             // attention weight of the point
    float ds;            // gradient of its logit
};


// MODE: BWD_FUSED = the whole chain; BWD_AV = backward of deform_av alone (`attn` given, dA written to `ddense`'s place
// is not needed: it goes to `grad_attn`, no logit gradients); BWD_QK = backward of deform_qk alone (`attn` carries the
// logit gradients dS, no aggregation part).
constexpr int BWD_FUSED = 0, BWD_AV = 1, BWD_QK = 2;

// In the form of deform_window_kernel (see there): the points of a pixel side by side, without branches, each point's place in the windows kept from
// pass to pass, a block = pixels of one (image, group).  The two windows of a thread (D and dWd going in, dD and Wd coming out) share its two
// columns of shared memory.  Points outside the window are few and hold up their warp, which gathers them together, a channel to a
// lane, while they are; each thread its own where there are many (lines at 40 or none: slower).  8 x 4 groups x 128x128 pixels, 9 points, float32 |
// bfloat16, us: sigma 0.5 118 -> 76 | 114 -> 74 (branches on each point before, in which one far point held its block), 1.0 1209 -> 418 |
// 1183 -> 450, 1.5 855 -> 673 | 865 -> 763; 1 point 108 -> 46 | 93 -> 42, 16 points 257 -> 240 | 267 -> 201.  Bound by latency at 16 warps per SM
// (128 registers, of which the form for 9 points spills 60).
template <typename T, int PMAX, int MODE>
__global__ void __launch_bounds__(WIN_THREADS, 4)
deform_window_bwd_kernel(const T *grad_out, const T *value, const T *offset,
                         const T *attn, const float *dense /* D [B*G, 25, hi] */,
                         const float *dwin /* dWd [B*G, 25, hi] */, T *ddense /* dD, out */,
                         T *window /* Wd, out */, T *grad_offset, T *grad_attn /* BWD_AV only */,
                         OutlierGrad *taps,
                         unsigned int *tap_count, int B, int C, int H, int W, int P_runtime, int G) {
    begin_after_previous();
    __shared__ float sd[MODE != BWD_AV ? 25 : 1][WIN_THREADS], sw[MODE != BWD_QK ? 25 : 1][WIN_THREADS];
    constexpr int MANY = 16;      // points outside the window of a warp's pixels
    const int P = PMAX == 9 ? 9 : P_runtime;
    const unsigned sW = 2 * W;
    const int gc = C / G;
    const size_t hi = (size_t)(2 * H) * sW, lo = (size_t)H * W;
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    const unsigned blocks = ((unsigned)hi + blockDim.x - 1) / blockDim.x, groups = (unsigned)(B * G);      // of an (image, group)
    float *const dcol = &sd[0][tid], *const wcol = &sw[0][tid];
    for (unsigned bg = blockIdx.y; bg < groups; bg += gridDim.y)
    for (unsigned block = blockIdx.x; block < blocks; block += gridDim.x) {
        const unsigned at_pix = block * blockDim.x + tid, pix = at_pix < hi ? at_pix : 0u;
        const bool live = at_pix < hi;
        const int qh = (int)(pix / sW), qw = (int)(pix - (unsigned)qh * sW), py = qh >> 1, px = qw >> 1;
        const T *offp = offset + (size_t)bg * P * 2 * hi + pix, *ap = attn + (size_t)bg * P * hi + pix;
        const float *dp = dense + (size_t)bg * 25 * hi + pix, *wp = dwin + (size_t)bg * 25 * hi + pix;
#pragma unroll
        for (int k = 0; k < 25; ++k) {
            if (MODE != BWD_AV) dcol[k * WIN_THREADS] = live ? __ldcs(dp + (size_t)k * hi) : 0.f;
            if (MODE != BWD_QK) wcol[k * WIN_THREADS] = live ? __ldcs(wp + (size_t)k * hi) : 0.f;
        }
        WindowPoints<PMAX> pts;
        pts.load(offp, hi, live, P);
        float at[PMAX];
#pragma unroll
        for (int p = 0; p < PMAX; ++p) at[p] = live && p < P ? to_acc(ap[(size_t)p * hi]) : 0.f;
        // ---- pass 1: dA_p and the bilinear forms of the offset gradients: value (1-lh, lh) x (1-lw, lw); d/dh (-1, 1) x (1-lw, lw); d/dw (1-lh, lh) x (-1, 1)
        float da[PMAX], gh1[PMAX], gw1[PMAX], gh2[PMAX], gw2[PMAX];
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            pts.set(p, live && p < P, H, W, py, px);
            const bool in = pts.dense >> p & 1;
            const float lh = pts.lh[p], lw = pts.lw[p], hh = 1.f - lh, hw = 1.f - lw;
            da[p] = gh1[p] = gw1[p] = gh2[p] = gw2[p] = 0.f;
            if (MODE != BWD_QK) {
                const float *c = wcol + pts.at(p);
                const float w00 = c[0], w01 = c[WIN_THREADS], w10 = c[5 * WIN_THREADS], w11 = c[6 * WIN_THREADS];
                const float top = hw * w00 + lw * w01, bot = hw * w10 + lw * w11;
                da[p] = in ? hh * top + lh * bot : 0.f;
                gh1[p] = in ? bot - top : 0.f;
                gw1[p] = in ? (hh * w01 + lh * w11) - (hh * w00 + lh * w10) : 0.f;
            }
            if (MODE != BWD_AV) {
                const float *c = dcol + pts.at(p);
                const float d00 = c[0], d01 = c[WIN_THREADS], d10 = c[5 * WIN_THREADS], d11 = c[6 * WIN_THREADS];
                gh2[p] = in ? (hw * d10 + lw * d11) - (hw * d00 + lw * d01) : 0.f;
                gw2[p] = in ? (hh * d01 + lh * d11) - (hh * d00 + lh * d10) : 0.f;
            }
        }
        if (MODE != BWD_QK) {         // dA of the points outside the window
            const T *gp = grad_out + (size_t)bg * gc * hi, *vp = value + (size_t)bg * gc * lo;
            const unsigned few = __reduce_add_sync(0xffffffffu, (unsigned)__popc(pts.outliers));
            if (few > MANY) {
                for (unsigned left = pts.outliers; left != 0; left &= left - 1) {
                    const int p = __ffs(left) - 1;
                    Bilinear<float> bl;
                    bl.setup(float(py) + to_acc(offp[(size_t)(2 * p + 1) * hi]), float(px) + to_acc(offp[(size_t)(2 * p) * hi]), H, W);
                    float acc = 0.f;
                    const T *v0 = vp, *g0 = gp + pix;             // pointers that advance: with products of the channel the loop takes half as long again
#pragma unroll 4
                    for (int c = 0; c < gc; ++c, v0 += lo, g0 += hi) acc += bl.sample(v0) * to_acc(*g0);
                    put(da, p, acc);
                }
            } else {
                for (unsigned lanes = __ballot_sync(0xffffffffu, pts.outliers != 0); lanes != 0; lanes &= lanes - 1) {
                    const int src = __ffs(lanes) - 1;
                    const unsigned spix = __shfl_sync(0xffffffffu, pix, src);
                    const int sh = (int)(spix / sW), spy = sh >> 1, spx = (int)(spix - (unsigned)sh * sW) >> 1;
                    const T *so = offset + (size_t)bg * P * 2 * hi + spix;
                    for (unsigned left = __shfl_sync(0xffffffffu, pts.outliers, src); left != 0; left &= left - 1) {
                        const int p = __ffs(left) - 1;
                        Bilinear<float> bl;
                        bl.setup(float(spy) + to_acc(so[(size_t)(2 * p + 1) * hi]), float(spx) + to_acc(so[(size_t)(2 * p) * hi]), H, W);
                        float acc = 0.f;
                        for (int c = lane; c < gc; c += 32) acc += bl.sample(vp + (size_t)c * lo) * to_acc(gp[(size_t)c * hi + spix]);
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                        if (lane == src) put(da, p, acc);
                    }
                }
            }
        }
        float dot = 0.f;
#pragma unroll
        for (int p = 0; p < PMAX; ++p) dot += at[p] * da[p];
        // ---- pass 2: logit gradients, dD, Wd (the two shared windows become the accumulators), offset gradients
#pragma unroll
        for (int k = 0; k < 25; ++k) {
            if (MODE != BWD_AV) dcol[k * WIN_THREADS] = 0.f;
            if (MODE != BWD_QK) wcol[k * WIN_THREADS] = 0.f;
        }
        T *gop = grad_offset + (size_t)bg * P * 2 * hi + pix;
#pragma unroll
        for (int p = 0; p < PMAX; ++p) {
            const bool on = live && p < P, in = pts.dense >> p & 1;
            // BWD_QK: `attn` holds the logit gradients themselves; BWD_AV: no logit gradient, dA goes out as it is
            const float a = MODE == BWD_QK ? 0.f : at[p], ds = MODE == BWD_QK ? at[p] : MODE == BWD_AV ? 0.f : a * (da[p] - dot);
            if (MODE == BWD_AV && on) grad_attn[((size_t)bg * P + p) * hi + pix] = from_acc<T>(da[p]);
            da[p] = ds;
            const float lh = pts.lh[p], lw = pts.lw[p], hw = 1.f - lw;
            if (MODE != BWD_AV) {
                float *c = dcol + pts.at(p);
                const float add = in ? ds : 0.f, t = add * (1.f - lh), u = add * lh;
                const float c00 = c[0], c01 = c[WIN_THREADS], c10 = c[5 * WIN_THREADS], c11 = c[6 * WIN_THREADS];
                c[0] = c00 + t * hw; c[WIN_THREADS] = c01 + t * lw; c[5 * WIN_THREADS] = c10 + u * hw; c[6 * WIN_THREADS] = c11 + u * lw;
            }
            if (MODE != BWD_QK) {
                float *c = wcol + pts.at(p);
                const float add = in ? a : 0.f, t = add * (1.f - lh), u = add * lh;
                const float c00 = c[0], c01 = c[WIN_THREADS], c10 = c[5 * WIN_THREADS], c11 = c[6 * WIN_THREADS];
                c[0] = c00 + t * hw; c[WIN_THREADS] = c01 + t * lw; c[5 * WIN_THREADS] = c10 + u * hw; c[6 * WIN_THREADS] = c11 + u * lw;
            }
            if (on && !(pts.outliers >> p & 1)) {      // the list kernel writes the offset gradients of the outliers
                gop[(size_t)(2 * p) * hi] = from_acc<T>(a * gw1[p] + ds * gw2[p]);
                gop[(size_t)(2 * p + 1) * hi] = from_acc<T>(a * gh1[p] + ds * gh2[p]);
            }
        }
        if (live) {
            T *ddp = ddense + (size_t)bg * 25 * hi + pix, *wdp = window + (size_t)bg * 25 * hi + pix;
#pragma unroll
            for (int k = 0; k < 25; ++k) {
                if (MODE != BWD_AV) ddp[(size_t)k * hi] = from_acc<T>(dcol[k * WIN_THREADS]);
                if (MODE != BWD_QK) wdp[(size_t)k * hi] = from_acc<T>(wcol[k * WIN_THREADS]);
            }
        }
        const unsigned int any = __ballot_sync(0xffffffffu, pts.outliers != 0);
        if (any != 0) {
            const int mine = __popc(pts.outliers);
            int incl = mine;
#pragma unroll
            for (int sft = 1; sft < 32; sft <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, sft);
                if (lane >= sft) incl += up;
            }
            const int warp_total = __shfl_sync(0xffffffffu, incl, 31);
            unsigned int base = 0;
            if (lane == 0) base = atomicAdd(tap_count, (unsigned int)warp_total);
            base = __shfl_sync(0xffffffffu, base, 0);
            unsigned int pos = base + (unsigned int)(incl - mine);
#pragma unroll
            for (int p = 0; p < PMAX; ++p)
                if (pts.outliers >> p & 1) {
                    OutlierGrad t;
                    t.k = (unsigned int)(bg * P + p); t.pix = pix; t.a = MODE == BWD_QK ? 0.f : at[p]; t.ds = da[p];
                    taps[pos++] = t;
                }
        }
    }
}

// Gradients of the listed outlier points: SUB threads per point share its sampling set-up and take every SUB-th
// channel; dQ, dKey and dV are added to what the SAPA-B kernels wrote (atomics), the point's offset gradient is written.
// TA = type of the scatter targets grad_key / grad_value: T itself in float32; float for 16-bit tensors, where they are
// zeroed side buffers that deform_add_scatter_kernel folds into the 16-bit gradients afterwards (a 16-bit atomic per
// corner and channel was 2x slower than the whole float32 pass and rounds at every addition).
template <int SUB, typename T, typename TA>
__device__ __forceinline__ void outlier_points_bwd(const OutlierGrad *taps, unsigned int n,
                                          const T *grad_out, const T *query, const T *key,
                                          const T *value, const T *offset, T *grad_query,
                                          TA *grad_key, TA *grad_value, T *grad_offset,
                                          int Cq, int C, int H, int W, int P, int G) {
    const int sW = 2 * W, gq = Cq / G, gc = C / G;
    const size_t hi = (size_t)(2 * H) * sW, lo = (size_t)H * W;
    const int lane = threadIdx.x & 31, sub = lane % SUB;
    const unsigned int group_mask = SUB == 32 ? 0xffffffffu : 0xffu << (lane & ~7);
    // entries of a short list are spread over the blocks, those of a long one stay next to their neighbours
    const unsigned int first = SUB == 32 ? threadIdx.x / SUB * gridDim.x + blockIdx.x : (blockIdx.x * blockDim.x + threadIdx.x) / SUB;
    for (unsigned int e = first; e < n; e += gridDim.x * blockDim.x / SUB) {
        const OutlierGrad t = taps[e];
        const size_t pix = t.pix;
        const int px = (int)(pix % sW) >> 1, py = (int)(pix / sW) >> 1;
        const float w = float(px) + to_acc(offset[(size_t)t.k * 2 * hi + pix]);
        const float h = float(py) + to_acc(offset[(size_t)t.k * 2 * hi + hi + pix]);
        Bilinear<float> bl;
        bl.setup(h, w, H, W);
        const float hh = 1.f - bl.lh, hw = 1.f - bl.lw;
        const size_t bg = t.k / (unsigned int)P;
        float g_w = 0.f, g_h = 0.f;
        for (int c = sub; c < gc && grad_value != nullptr; c += SUB) {      // aggregation: dV scatter and its offset gradient
            float v00, v01, v10, v11;
            bl.corners(value + (bg * gc + c) * lo, v00, v01, v10, v11);
            const float tw = to_acc(grad_out[(bg * gc + c) * hi + pix]) * t.a;
            TA *gp = grad_value + (bg * gc + c) * lo;
            if (bl.i00 >= 0) atomicAdd(gp + bl.i00, from_acc<TA>(bl.w00 * tw));
            if (bl.i01 >= 0) atomicAdd(gp + bl.i01, from_acc<TA>(bl.w01 * tw));
            if (bl.i10 >= 0) atomicAdd(gp + bl.i10, from_acc<TA>(bl.w10 * tw));
            if (bl.i11 >= 0) atomicAdd(gp + bl.i11, from_acc<TA>(bl.w11 * tw));
            g_w += (-hh * v00 + hh * v01 - bl.lh * v10 + bl.lh * v11) * tw;
            g_h += (-hw * v00 - bl.lw * v01 + hw * v10 + bl.lw * v11) * tw;
        }
        for (int c = sub; c < gq && grad_query != nullptr; c += SUB) {      // similarity: dQ, dKey scatter and its offset gradient
            float v00, v01, v10, v11;
            bl.corners(key + (bg * gq + c) * lo, v00, v01, v10, v11);
            atomicAdd(grad_query + (bg * gq + c) * hi + pix, from_acc<T>(t.ds * (bl.w00 * v00 + bl.w01 * v01 + bl.w10 * v10 + bl.w11 * v11)));
            const float tw = t.ds * to_acc(query[(bg * gq + c) * hi + pix]);
            TA *gp = grad_key + (bg * gq + c) * lo;
            if (bl.i00 >= 0) atomicAdd(gp + bl.i00, from_acc<TA>(bl.w00 * tw));
            if (bl.i01 >= 0) atomicAdd(gp + bl.i01, from_acc<TA>(bl.w01 * tw));
            if (bl.i10 >= 0) atomicAdd(gp + bl.i10, from_acc<TA>(bl.w10 * tw));
            if (bl.i11 >= 0) atomicAdd(gp + bl.i11, from_acc<TA>(bl.w11 * tw));
            g_w += (-hh * v00 + hh * v01 - bl.lh * v10 + bl.lh * v11) * tw;
            g_h += (-hw * v00 - bl.lw * v01 + hw * v10 + bl.lw * v11) * tw;
        }
#pragma unroll
        for (int sh = 1; sh < SUB; sh <<= 1) {
            g_w += __shfl_xor_sync(group_mask, g_w, sh);
            g_h += __shfl_xor_sync(group_mask, g_h, sh);
        }
        if (sub == 0) {
            grad_offset[(size_t)t.k * 2 * hi + pix] = from_acc<T>(g_w);
            grad_offset[(size_t)t.k * 2 * hi + hi + pix] = from_acc<T>(g_h);
        }
    }
}

template <typename T, typename TA>      // a warp per entry of a short list, as in the forward pass
__global__ void deform_outlier_bwd_kernel(const OutlierGrad *taps, const unsigned int *tap_count,
                                          const T *grad_out, const T *query, const T *key,
                                          const T *value, const T *offset, T *grad_query,
                                          TA *grad_key, TA *grad_value, T *grad_offset,
                                          int Cq, int C, int H, int W, int P, int G) {
    begin_after_previous();
    const unsigned int n = *tap_count;
    if (n <= gridDim.x * (blockDim.x / 32))
        outlier_points_bwd<32>(taps, n, grad_out, query, key, value, offset, grad_query, grad_key, grad_value, grad_offset, Cq, C, H, W, P, G);
    else
        outlier_points_bwd<8>(taps, n, grad_out, query, key, value, offset, grad_query, grad_key, grad_value, grad_offset, Cq, C, H, W, P, G);
}

// The float32 side buffers of the 16-bit gradients: zeroed before the list kernel, added to the gradients after it (one rounding per
// element).  A short list touches a few thousand of the buffers' cells: those alone are zeroed, and taken back by an exchange that
// gives each cell's whole sum to one of the points that share it.  A long list goes over the buffers (42 MB at 8 images of 320
// channels, 64 x 64: 10 + 26 us; the short form, for 582 points: 5 + 10 us).
struct Scatter { float *key, *value; size_t n_key, n_value; int gq, gc; };      // the value buffer lies behind the key buffer

// f(cell index of the key buffer or of the value buffer, which) for the four corners of every listed point and all channels of its
// group; a warp per corner
template <typename T, typename F>
__device__ __forceinline__ void for_scattered(const OutlierGrad *taps, unsigned int n, const T *offset, const Scatter &sc, int H, int W,
                                              int P, F f) {
    const int sW = 2 * W;
    const size_t hi = (size_t)(2 * H) * sW, lo = (size_t)H * W;
    for (unsigned int e = threadIdx.x / 32 * gridDim.x + blockIdx.x; e < 4 * n; e += gridDim.x * (blockDim.x / 32)) {
        const OutlierGrad t = taps[e >> 2];
        const size_t pix = t.pix, bg = t.k / (unsigned int)P;
        const int px = (int)(pix % sW) >> 1, py = (int)(pix / sW) >> 1;
        const float w = float(px) + to_acc(offset[(size_t)t.k * 2 * hi + pix]), h = float(py) + to_acc(offset[(size_t)t.k * 2 * hi + hi + pix]);
        Bilinear<float> bl;
        bl.setup(h, w, H, W);
        const int at = (e & 2) != 0 ? ((e & 1) != 0 ? bl.i11 : bl.i10) : (e & 1) != 0 ? bl.i01 : bl.i00;
        if (at < 0) continue;
        for (int c = threadIdx.x & 31; c < sc.gq + sc.gc; c += 32) {
            const bool key = c < sc.gq;
            f((key ? bg * sc.gq + c : bg * sc.gc + (c - sc.gq)) * lo + at, key);
        }
    }
}

template <typename T>
__global__ void deform_zero_scatter_kernel(const OutlierGrad *taps, const unsigned int *tap_count, const T *offset,
                                           const Scatter sc, int H, int W, int P) {
    begin_after_previous();
    const unsigned int n = *tap_count;
    if (n <= gridDim.x * (blockDim.x / 32)) {
        for_scattered(taps, n, offset, sc, H, W, P, [&](size_t i, bool key) { (key ? sc.key : sc.value)[i] = 0.f; });
        return;
    }
    float *base = sc.n_key != 0 ? sc.key : sc.value;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < sc.n_key + sc.n_value; i += (size_t)gridDim.x * blockDim.x) base[i] = 0.f;
}

template <typename T>
__global__ void deform_add_scatter_kernel(const OutlierGrad *taps, const unsigned int *tap_count, const T *offset,
                                          const Scatter sc, T *grad_key, T *grad_value, int H, int W, int P) {
    begin_after_previous();
    const unsigned int n = *tap_count;
    if (n <= gridDim.x * (blockDim.x / 32)) {
        for_scattered(taps, n, offset, sc, H, W, P, [&](size_t i, bool key) {
            const float v = atomicExch((key ? sc.key : sc.value) + i, 0.f);
            T *dst = (key ? grad_key : grad_value) + i;
            if (v != 0.f) *dst = from_acc<T>(to_acc(*dst) + v);
        });
        return;
    }
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < sc.n_key + sc.n_value; i += stride) {
        if (i < sc.n_key) grad_key[i] = from_acc<T>(to_acc(grad_key[i]) + sc.key[i]);
        else grad_value[i - sc.n_key] = from_acc<T>(to_acc(grad_value[i - sc.n_key]) + sc.value[i - sc.n_key]);
    }
}

// ---------------------------------------------------------------------------------- backward, fused
// Gradients of out = deform_av(softmax_p(deform_qk(q, k, off)), v, off) in ONE kernel.  One thread per (image, group,
// high-res pixel) walks the P points three times, with the per-point values parked in shared memory:
//   pass A (aggregation):  dA_p = sum_c dOut_c * val_c(p);  dV_c[corner] += w * dOut_c * A_p (atomic scatter);
//                          offset gradient of the aggregation;
//   pass B (softmax):      dS_p = A_p * (dA_p - sum_q A_q dA_q);
//   pass C (similarity):   dQ_c = sum_p dS_p * val_c(p) (this thread is the only writer: plain stores, deterministic);
//                          dKey_c[corner] += w * dS_p * Q_c (atomic scatter); offset gradient of the similarity.
// The two offset gradients are added here, so the offsets and the attention map are read once and no intermediate
// tensor ([B,G,P,sH,sW] attention gradient, logit gradient, second offset gradient) ever reaches HBM.
template <typename T, int NTHR>
__global__ void __launch_bounds__(NTHR)
deform_fused_bwd_kernel(const T *__restrict__ grad_out, const T *__restrict__ query, const T *__restrict__ key,
                        const T *__restrict__ value, const T *__restrict__ offset, const T *__restrict__ attn,
                        typename AccOf<T>::type *__restrict__ grad_query, typename AccOf<T>::type *__restrict__ grad_key,
                        typename AccOf<T>::type *__restrict__ grad_value, T *__restrict__ grad_offset,
                        int B, int Cq, int C, int H, int W, int P, int s, int G) {
    using A = typename AccOf<T>::type;
    __shared__ A s_h[MAXP][NTHR], s_w[MAXP][NTHR], s_d[MAXP][NTHR], s_gw[MAXP][NTHR], s_gh[MAXP][NTHR];
    const int sH = s * H, sW = s * W, AC = G * P, gq = Cq / G, gc = C / G;
    const size_t hi = (size_t)sH * sW, lo = (size_t)H * W;
    const int tx = threadIdx.x;
    const long long total = (long long)B * G * hi;
    for (long long i = blockIdx.x * (long long)NTHR + tx; i < total; i += (long long)gridDim.x * NTHR) {
        const size_t pix = (size_t)(i % hi);
        const int qw = (int)(pix % sW), qh = (int)(pix / sW);
        const int g = (int)((i / hi) % G);
        const int b = (int)(i / (hi * G));
        const size_t k0 = (size_t)b * AC + (size_t)g * P;              // first (group, point) plane of this thread
        const T *ap = attn + k0 * hi + pix;
        // ---- pass A
        A dot = 0;
        for (int p = 0; p < P; ++p) {
            const A w = A(qw / s) + to_acc(offset[(k0 + p) * 2 * hi + pix]);
            const A h = A(qh / s) + to_acc(offset[(k0 + p) * 2 * hi + hi + pix]);
            Bilinear<A, true> bl;
            bl.setup(h, w, H, W);
            A dA = 0, g_w = 0, g_h = 0;
            if (bl.inside) {
                const A hh = A(1) - bl.lh, hw = A(1) - bl.lw;
                const A a_p = to_acc(ap[(size_t)p * hi]);
                const size_t ch0 = (size_t)b * C + (size_t)g * gc;
                for (int c = 0; c < gc; ++c) {
                    A v00, v01, v10, v11;
                    bl.corners(value + (ch0 + c) * lo, v00, v01, v10, v11);
                    const A t = to_acc(grad_out[(ch0 + c) * hi + pix]);
                    dA += t * (bl.w00 * v00 + bl.w01 * v01 + bl.w10 * v10 + bl.w11 * v11);
                    const A tw = t * a_p;
                    A *gp = grad_value + (ch0 + c) * lo;
                    if (bl.i00 >= 0) atomic_add(gp + bl.i00, bl.w00 * tw);
                    if (bl.i01 >= 0) atomic_add(gp + bl.i01, bl.w01 * tw);
                    if (bl.i10 >= 0) atomic_add(gp + bl.i10, bl.w10 * tw);
                    if (bl.i11 >= 0) atomic_add(gp + bl.i11, bl.w11 * tw);
                    g_w += (-hh * v00 + hh * v01 - bl.lh * v10 + bl.lh * v11) * tw;
                    g_h += (-hw * v00 - bl.lw * v01 + hw * v10 + bl.lw * v11) * tw;
                }
                dot += a_p * dA;
            }
            s_h[p][tx] = h; s_w[p][tx] = w; s_d[p][tx] = dA; s_gw[p][tx] = g_w; s_gh[p][tx] = g_h;
        }
        // ---- pass B + C
        const size_t qch0 = (size_t)b * Cq + (size_t)g * gq;
        for (int p = 0; p < P; ++p) {
            const A dS = to_acc(ap[(size_t)p * hi]) * (s_d[p][tx] - dot);
            Bilinear<A, true> bl;
            bl.setup(s_h[p][tx], s_w[p][tx], H, W);
            A g_w = s_gw[p][tx], g_h = s_gh[p][tx];
            const bool first = p == 0;
            if (bl.inside) {
                const A hh = A(1) - bl.lh, hw = A(1) - bl.lw;
                for (int c = 0; c < gq; ++c) {
                    A v00, v01, v10, v11;
                    bl.corners(key + (qch0 + c) * lo, v00, v01, v10, v11);
                    const A val = bl.w00 * v00 + bl.w01 * v01 + bl.w10 * v10 + bl.w11 * v11;
                    A *qg = grad_query + (qch0 + c) * hi + pix;
                    *qg = first ? dS * val : *qg + dS * val;
                    const A tw = dS * to_acc(query[(qch0 + c) * hi + pix]);
                    A *gp = grad_key + (qch0 + c) * lo;
                    if (bl.i00 >= 0) atomic_add(gp + bl.i00, bl.w00 * tw);
                    if (bl.i01 >= 0) atomic_add(gp + bl.i01, bl.w01 * tw);
                    if (bl.i10 >= 0) atomic_add(gp + bl.i10, bl.w10 * tw);
                    if (bl.i11 >= 0) atomic_add(gp + bl.i11, bl.w11 * tw);
                    g_w += (-hh * v00 + hh * v01 - bl.lh * v10 + bl.lh * v11) * tw;
                    g_h += (-hw * v00 - bl.lw * v01 + hw * v10 + bl.lw * v11) * tw;
                }
            } else if (first) {
                for (int c = 0; c < gq; ++c) grad_query[(qch0 + c) * hi + pix] = A(0);
            }
            grad_offset[(k0 + p) * 2 * hi + pix] = from_acc<T>(g_w);
            grad_offset[(k0 + p) * 2 * hi + hi + pix] = from_acc<T>(g_h);
        }
    }
}

static inline int grid_1d(long long total, int threads) {
    long long blocks = (total + threads - 1) / threads;
    const long long cap = 148LL * 64;
    return (int)(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}

// The window kernels for up to 4, 8, 9 (exactly) or 16 points: their loops run over all points of the instance side by side, so that those
// that are not there cost what the others do.  8 x 4 groups x 128x128 pixels, with one point, the forms of 16 and 4 points: fused op
// float32 189 and 141 us, bfloat16 148 and 102; 16 points 223 and 176.
template <typename F> static void for_points(int P, F launch) {
    if (P <= 4) launch(std::integral_constant<int, 4>());
    else if (P <= 8) launch(std::integral_constant<int, 8>());
    else if (P == 9) launch(std::integral_constant<int, 9>());
    else launch(std::integral_constant<int, MAXP>());
}
// Blocks: pixels of an (image, group) along x, the (image, group)s along y; half-sized ones where the last of a small image would be
// half empty or more (2048 x 4 groups of 4x16 pixels, float32: forward 211 us with whole blocks, 197 with halves; forward and backward 738 and 719,
// bfloat16 605 and 576).
static unsigned window_threads(size_t hi) { return hi <= 4 * WIN_THREADS && (hi - 1) % WIN_THREADS < WIN_THREADS / 2 ? WIN_THREADS / 2 : WIN_THREADS; }
static dim3 window_grid(size_t hi, unsigned threads, int groups) { return dim3((unsigned)((hi + threads - 1) / threads), (unsigned)(groups < 65535 ? groups : 65535), 1); }
template <int MODE, typename T, typename... A> static void launch_window(int P, int groups, size_t hi, cudaStream_t st, A... args) {
    const unsigned threads = window_threads(hi);
    for_points(P, [&](auto most) { launch_next(deform_window_kernel<T, decltype(most)::value, MODE>, window_grid(hi, threads, groups), threads, 0, st, args...); });
}

template <int MODE, typename T, typename... A> static void launch_window_bwd(int P, int groups, size_t hi, cudaStream_t st, A... args) {
    const unsigned threads = window_threads(hi);
    for_points(P, [&](auto most) { launch_in_order(deform_window_bwd_kernel<T, decltype(most)::value, MODE>, window_grid(hi, threads, groups), threads, 0, st, args...); });
}

static int check_deform(const char *fn, int B, int Cq, int C, int H, int W, int P, int s, int G, int dtype) {
    SAPA_REQUIRE(B > 0 && Cq > 0 && C > 0 && H > 0 && W > 0, SAPA_ERR_ARGUMENT, "%s: sizes must be positive", fn);
    SAPA_REQUIRE(P >= 1, SAPA_ERR_ARGUMENT, "%s: num_point must be >= 1, got %d", fn, P);
    SAPA_REQUIRE(s >= 1, SAPA_ERR_ARGUMENT, "%s: scale_factor must be >= 1, got %d", fn, s);
    SAPA_REQUIRE(G >= 1 && Cq % G == 0 && C % G == 0, SAPA_ERR_ARGUMENT,
                 "%s: channels (%d, %d) must be divisible by groups (%d)", fn, Cq, C, G);
    SAPA_REQUIRE(dtype_size(dtype) != 0, SAPA_ERR_DTYPE, "%s: unknown dtype code %d", fn, dtype);
    SAPA_REQUIRE((long long)s * H * s * W < (1LL << 31), SAPA_ERR_ARGUMENT, "%s: image too large", fn);
    return SAPA_OK;
}


// The counter of the outlier list.  A kernel and not a memset: a memset between kernels keeps the ones around it from being set up
// ahead (float32 forward of 8 x 256 x 64x64 178.8 -> 174.0 us, its bfloat16 training 473 -> 455, with two such counters).
__global__ void deform_clear_counter_kernel(unsigned int *counter) {
    begin_after_previous();
    *counter = 0u;
}
static int clear_counter(const char *fn, unsigned int *counter, cudaStream_t st) {
    launch_next(deform_clear_counter_kernel, 1, 1, 0, st, counter);
    const cudaError_t e = cudaGetLastError();
    SAPA_REQUIRE(e == cudaSuccess, SAPA_ERR_LAUNCH, "%s: clearing the outlier counter failed: %s", fn, cudaGetErrorString(e));
    return SAPA_OK;
}

static int memset_async(void *p, size_t bytes, cudaStream_t st, const char *fn) {
    const cudaError_t e = cudaMemsetAsync(p, 0, bytes, st);
    SAPA_REQUIRE(e == cudaSuccess, SAPA_ERR_LAUNCH, "%s: cudaMemsetAsync failed: %s", fn, cudaGetErrorString(e));
    return SAPA_OK;
}

}  // namespace sapa

using namespace sapa;

extern "C" {

int sapa_deform_qk_forward(const void *query, const void *key, const void *offset, void *out, int B, int Cq, int H, int W,
                           int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_qk_forward";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, Cq, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, offset); SAPA_CHECK_PTR(fn, out);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return SAPA_DISPATCH_ALL(dtype, [&] {
        const long long total = (long long)B * G * P * s * H * s * W;
        deform_qk_fwd_kernel<scalar_t><<<grid_1d(total, 256), 256, 0, st>>>(
            static_cast<const scalar_t *>(query), static_cast<const scalar_t *>(key), static_cast<const scalar_t *>(offset),
            static_cast<scalar_t *>(out), B, Cq, H, W, P, s, G);
        return check_launch("deform_qk_fwd_kernel");
    });
}

int sapa_deform_av_forward(const void *attn, const void *value, const void *offset, void *out, int B, int C, int H, int W,
                           int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_av_forward";
    trace_reset();
    if (int e = check_deform(fn, B, C, C, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, attn); SAPA_CHECK_PTR(fn, value); SAPA_CHECK_PTR(fn, offset); SAPA_CHECK_PTR(fn, out);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return SAPA_DISPATCH_ALL(dtype, [&] {
        constexpr int CPT = 8;
        const int chunks = (C / G + CPT - 1) / CPT;
        const long long total = (long long)B * G * chunks * s * H * s * W;
        deform_av_fwd_kernel<scalar_t, CPT><<<grid_1d(total, 256), 256, 0, st>>>(
            static_cast<const scalar_t *>(attn), static_cast<const scalar_t *>(value), static_cast<const scalar_t *>(offset),
            static_cast<scalar_t *>(out), B, C, H, W, P, s, G);
        return check_launch("deform_av_fwd_kernel");
    });
}

int sapa_deform_fused_forward(const void *query, const void *key, const void *value, const void *offset, void *out,
                              void *attn, int B, int Cq, int C, int H, int W, int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_fused_forward";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, C, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, value); SAPA_CHECK_PTR(fn, offset);
    SAPA_CHECK_PTR(fn, out);
    SAPA_REQUIRE(P <= MAXP && dtype != SAPA_F64, SAPA_ERR_UNSUPPORTED,
                 "%s: no fused kernel for num_point=%d dtype=%d (use the separate ops)", fn, P, dtype);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return SAPA_DISPATCH_FAST(dtype, [&] {
        const int pix_blocks = ceil_div((long long)s * H * s * W, 32);
        const long long blocks = (long long)B * G * pix_blocks;
        if (blocks > 0x7fffffffLL) {
            set_error("too many blocks");
            return (int)SAPA_ERR_ARGUMENT;
        }
        deform_fused_fwd_kernel<scalar_t, 8><<<(unsigned)blocks, dim3(32, FY), 0, st>>>(
            static_cast<const scalar_t *>(query), static_cast<const scalar_t *>(key), static_cast<const scalar_t *>(value),
            static_cast<const scalar_t *>(offset), static_cast<scalar_t *>(out), static_cast<scalar_t *>(attn), B, Cq, C, H,
            W, P, s, G, pix_blocks);
        return check_launch("deform_fused_fwd_kernel");
    });
}

int sapa_deform_qk_backward(const void *grad_out, const void *query, const void *key, const void *offset, void *grad_query,
                            void *grad_key, void *grad_offset, int B, int Cq, int H, int W, int P, int s, int G, int dtype,
                            void *stream) {
    const char *fn = "sapa_deform_qk_backward";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, Cq, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, grad_out); SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, offset);
    SAPA_CHECK_PTR(fn, grad_query); SAPA_CHECK_PTR(fn, grad_key); SAPA_CHECK_PTR(fn, grad_offset);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t acc = dtype == SAPA_F64 ? 8 : 4;
    if (int e = memset_async(grad_query, (size_t)B * Cq * s * H * s * W * acc, st, fn)) return e;
    if (int e = memset_async(grad_key, (size_t)B * Cq * H * W * acc, st, fn)) return e;
    return SAPA_DISPATCH_ALL(dtype, [&] {
        using A = typename AccOf<scalar_t>::type;
        const long long total = (long long)B * G * P * s * H * s * W;
        deform_bwd_kernel<scalar_t, true><<<grid_1d(total, 256), 256, 0, st>>>(
            static_cast<const scalar_t *>(grad_out), static_cast<const scalar_t *>(query), static_cast<const scalar_t *>(key),
            static_cast<const scalar_t *>(offset), static_cast<A *>(grad_query), nullptr, static_cast<A *>(grad_key),
            static_cast<scalar_t *>(grad_offset), B, Cq, H, W, P, s, G);
        return check_launch("deform_bwd_kernel<qk>");
    });
}

int sapa_deform_av_backward(const void *grad_out, const void *attn, const void *value, const void *offset, void *grad_attn,
                            void *grad_value, void *grad_offset, int B, int C, int H, int W, int P, int s, int G, int dtype,
                            void *stream) {
    const char *fn = "sapa_deform_av_backward";
    trace_reset();
    if (int e = check_deform(fn, B, C, C, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, grad_out); SAPA_CHECK_PTR(fn, attn); SAPA_CHECK_PTR(fn, value); SAPA_CHECK_PTR(fn, offset);
    SAPA_CHECK_PTR(fn, grad_attn); SAPA_CHECK_PTR(fn, grad_value); SAPA_CHECK_PTR(fn, grad_offset);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t acc = dtype == SAPA_F64 ? 8 : 4;
    if (int e = memset_async(grad_value, (size_t)B * C * H * W * acc, st, fn)) return e;
    return SAPA_DISPATCH_ALL(dtype, [&] {
        using A = typename AccOf<scalar_t>::type;
        const long long total = (long long)B * G * P * s * H * s * W;
        deform_bwd_kernel<scalar_t, false><<<grid_1d(total, 256), 256, 0, st>>>(
            static_cast<const scalar_t *>(grad_out), static_cast<const scalar_t *>(attn), static_cast<const scalar_t *>(value),
            static_cast<const scalar_t *>(offset), nullptr, static_cast<scalar_t *>(grad_attn), static_cast<A *>(grad_value),
            static_cast<scalar_t *>(grad_offset), B, C, H, W, P, s, G);
        return check_launch("deform_bwd_kernel<av>");
    });
}

int sapa_deform_fused_backward(const void *grad_out, const void *query, const void *key, const void *value,
                               const void *offset, const void *attn, void *grad_query, void *grad_key, void *grad_value,
                               void *grad_offset, int B, int Cq, int C, int H, int W, int P, int s, int G, int dtype,
                               void *stream) {
    const char *fn = "sapa_deform_fused_backward";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, C, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, grad_out); SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, value);
    SAPA_CHECK_PTR(fn, offset); SAPA_CHECK_PTR(fn, attn); SAPA_CHECK_PTR(fn, grad_offset);
    SAPA_REQUIRE(grad_query != nullptr && grad_key != nullptr && grad_value != nullptr, SAPA_ERR_ARGUMENT,
                 "%s: a gradient buffer is NULL", fn);
    SAPA_REQUIRE(P <= MAXP, SAPA_ERR_UNSUPPORTED, "%s: no fused kernel for num_point=%d (use the separate ops)", fn, P);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t acc = dtype == SAPA_F64 ? 8 : 4;
    if (int e = memset_async(grad_key, (size_t)B * Cq * H * W * acc, st, fn)) return e;
    if (int e = memset_async(grad_value, (size_t)B * C * H * W * acc, st, fn)) return e;
    return SAPA_DISPATCH_ALL(dtype, [&] {
        using A = typename AccOf<scalar_t>::type;
        constexpr int NTHR = sizeof(A) == 8 ? 64 : 128;      // five per-point arrays of MAXP x NTHR accumulators in shared memory
        const long long total = (long long)B * G * s * H * s * W;
        deform_fused_bwd_kernel<scalar_t, NTHR><<<grid_1d(total, NTHR), NTHR, 0, st>>>(
            static_cast<const scalar_t *>(grad_out), static_cast<const scalar_t *>(query), static_cast<const scalar_t *>(key),
            static_cast<const scalar_t *>(value), static_cast<const scalar_t *>(offset), static_cast<const scalar_t *>(attn),
            static_cast<A *>(grad_query), static_cast<A *>(grad_key), static_cast<A *>(grad_value),
            static_cast<scalar_t *>(grad_offset), B, Cq, C, H, W, P, s, G);
        return check_launch("deform_fused_bwd_kernel");
    });
}

}  // extern "C"

// dispatchers of the SAPA-B logit and aggregation kernels (sapa_b.cu)
namespace sapa {
int run_sim(const void *hi, const void *lo, void *out, int B, int Cc, int H, int W, int K, int s, int dtype, cudaStream_t st, int groups);
int run_agg(const void *wt, const void *lo, void *out, int B, int Cc, int H, int W, int K, int s, int dtype, cudaStream_t st, int groups);
int run_gath(const void *hi, const void *wt, void *out, int B, int Cc, int H, int W, int K, int s, int dtype, cudaStream_t st, int groups);
int run_sim_slab(const void *hi, const void *lo, void *out, int B, int Cc, int H, int W, int rows, int top, int K, int s, int dtype,
                 cudaStream_t st, int groups);
int run_agg_slab(const void *wt, const void *lo, void *out, int B, int Cc, int H, int W, int rows, int top, int K, int s, int dtype,
                 cudaStream_t st, int groups);
int run_sim_mixed(const void *hi, const void *lo, float *out, int B, int Cc, int H, int W, int rows, int top, int dtype, cudaStream_t st, int groups);
bool fused_tma_supported(int W, int dtype);
}

extern "C" {

size_t sapa_deform_fused_forward_workspace(int B, int H, int W, int P, int s, int G, int dtype) {
    if (B <= 0 || H <= 0 || W <= 0 || P <= 0 || G <= 0 || s != 2) return 0;
    // 16-bit tensors: the mixed modes of the tensor-core kernels (16-bit operands, float32 windows).  Rows that are not multiples of 16 bytes run the
    // float32 chain on widened tensors, or the gather kernels, with float32 weights
    if (dtype != SAPA_F32 && !((dtype == SAPA_F16 || dtype == SAPA_BF16) && fused_tma_supported(W, dtype))) return 0;
    const size_t hi = (size_t)s * H * s * W;
    if ((size_t)B * G * hi >= 0xffffffffull) return 0;       // the outlier list indexes (image, group, pixel) with 32 bits
    // dense similarity + window weights (float32 whatever the tensors' type), the outlier list (worst case: every
    // point) and its counter
    return (size_t)B * G * 50 * hi * sizeof(float) + (size_t)B * G * hi * sizeof(OutlierTap) + 16;
}

int sapa_deform_fused_forward_slab(const void *query, const void *key, const void *value, const void *offset, void *out,
                                   void *attn, void *workspace, size_t workspace_bytes, int B, int Cq, int C, int H, int W,
                                   int halo_top, int halo_bottom, int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_fused_forward_slab";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, C, H, W, P, s, G, dtype)) return e;
    SAPA_REQUIRE(halo_top >= 0 && halo_bottom >= 0 && ((long long)halo_top + H + halo_bottom) * W < (1LL << 31), SAPA_ERR_ARGUMENT,
                 "%s: bad halo (%d, %d)", fn, halo_top, halo_bottom);
    const int rows = halo_top + H + halo_bottom;
    SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, value); SAPA_CHECK_PTR(fn, offset);
    SAPA_CHECK_PTR(fn, out);
    const size_t need = sapa_deform_fused_forward_workspace(B, H, W, P, s, G, dtype);
    SAPA_REQUIRE(s == 2 && P <= MAXP && need != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: the dense-window path needs s = 2, num_point <= %d and float32, or float16 / bfloat16 with rows of 16 bytes "
                 "(use sapa_deform_fused_forward)", fn, MAXP);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && aligned16(workspace), SAPA_ERR_WORKSPACE,
                 "%s: a 16-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    const size_t hi = (size_t)s * H * s * W;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the window weights have the tensors' type (the aggregation kernel rounds them to it anyway), the similarity is
    // always float32; both regions are sized for float32
    float *dense = static_cast<float *>(workspace);
    void *window = dense + (size_t)B * G * 25 * hi;
    OutlierTap *taps = reinterpret_cast<OutlierTap *>(dense + (size_t)B * G * 50 * hi);
    unsigned int *tap_count = reinterpret_cast<unsigned int *>(taps + (size_t)B * G * hi);
    if (int e = clear_counter(fn, tap_count, st)) return e;
    // 1. dense 25-slot similarity of every group: the B x G groups are images of Cq / G channels.  16-bit tensors: the
    //    logits leave the tensor-core kernel as float32 (a 16-bit logit would cost the softmax two digits)
    if (dtype == SAPA_F32) {
        if (int e = run_sim_slab(query, key, dense, B * G, Cq / G, H, W, rows, halo_top, 5, 2, dtype, st, G)) return e;
    } else {
        if (int e = run_sim_mixed(query, key, dense, B * G, Cq / G, H, W, rows, halo_top, dtype, st, G)) return e;
    }
    // 2. attention over the points, dense window weights, list of the points that leave the window
    {
        const int e = SAPA_DISPATCH_FAST(dtype, [&] {
            launch_window<WIN_FUSED, scalar_t>(P, B * G, hi, st, static_cast<const scalar_t *>(query), static_cast<const scalar_t *>(key),
                                               static_cast<const scalar_t *>(offset), dense, static_cast<scalar_t *>(attn), static_cast<scalar_t *>(window), taps,
                                               tap_count, B, Cq, H, W, P, G, rows, halo_top);
            return check_launch("deform_window_kernel");
        });
        if (e) return e;
    }
    // 3. aggregation of every group's channels over the window
    if (int e = run_agg_slab(window, value, out, B * G, C / G, H, W, rows, halo_top, 5, 2, dtype, st, G)) return e;
    // 4. the listed points (the count is only known on the device: a fixed grid strides over the list)
    return SAPA_DISPATCH_FAST(dtype, [&] {
        launch_next_with_l1(deform_outlier_kernel<scalar_t>, 148 * 8, 256, st, taps, tap_count, static_cast<const scalar_t *>(value),
                                                                 static_cast<const scalar_t *>(offset), static_cast<scalar_t *>(out),
                                                                 C, H, W, P, G, rows, halo_top);
        return check_launch("deform_outlier_kernel");
    });
}

int sapa_deform_fused_forward_dense(const void *query, const void *key, const void *value, const void *offset, void *out,
                                    void *attn, void *workspace, size_t workspace_bytes, int B, int Cq, int C, int H, int W,
                                    int P, int s, int G, int dtype, void *stream) {
    return sapa_deform_fused_forward_slab(query, key, value, offset, out, attn, workspace, workspace_bytes, B, Cq, C, H, W, 0, 0,
                                          P, s, G, dtype, stream);
}

// deform_qk and deform_av through the dense window (s = 2, float32): the halves of the fused forward, with the reference's
// op boundaries (raw logits out / attention in).  Workspace as for sapa_deform_fused_forward_dense.
int sapa_deform_qk_forward_dense(const void *query, const void *key, const void *offset, void *out, void *workspace,
                                 size_t workspace_bytes, int B, int Cq, int H, int W, int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_qk_forward_dense";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, Cq, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, offset); SAPA_CHECK_PTR(fn, out);
    const size_t need = sapa_deform_fused_forward_workspace(B, H, W, P, s, G, dtype);
    SAPA_REQUIRE(s == 2 && P <= MAXP && need != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: the dense-window path needs s = 2, num_point <= %d and float32, or float16 / bfloat16 with rows of 16 bytes "
                 "(use sapa_deform_qk_forward)", fn, MAXP);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && aligned16(workspace), SAPA_ERR_WORKSPACE,
                 "%s: a 16-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    const size_t hi = (size_t)s * H * s * W;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float *dense = static_cast<float *>(workspace);
    if (dtype == SAPA_F32) {
        if (int e = run_sim(query, key, dense, B * G, Cq / G, H, W, 5, 2, dtype, st, G)) return e;
    } else {
        if (int e = run_sim_mixed(query, key, dense, B * G, Cq / G, H, W, H, 0, dtype, st, G)) return e;
    }
    return SAPA_DISPATCH_FAST(dtype, [&] {
        for_points(P, [&](auto most) {
            launch_next(deform_logits_kernel<scalar_t, decltype(most)::value>, grid_1d((long long)B * G * hi, WIN_THREADS), WIN_THREADS, 0, st,
                        static_cast<const scalar_t *>(query), static_cast<const scalar_t *>(key), static_cast<const scalar_t *>(offset), dense,
                        static_cast<scalar_t *>(out), B * G, Cq / G, H, W, P);
        });
        return check_launch("deform_window_kernel<logits>");
    });
}

int sapa_deform_av_forward_dense(const void *attn, const void *value, const void *offset, void *out, void *workspace,
                                 size_t workspace_bytes, int B, int C, int H, int W, int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_av_forward_dense";
    trace_reset();
    if (int e = check_deform(fn, B, C, C, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, attn); SAPA_CHECK_PTR(fn, value); SAPA_CHECK_PTR(fn, offset); SAPA_CHECK_PTR(fn, out);
    const size_t need = sapa_deform_fused_forward_workspace(B, H, W, P, s, G, dtype);
    SAPA_REQUIRE(s == 2 && P <= MAXP && need != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: the dense-window path needs s = 2, num_point <= %d and float32, or float16 / bfloat16 with rows of 16 bytes "
                 "(use sapa_deform_av_forward)", fn, MAXP);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && aligned16(workspace), SAPA_ERR_WORKSPACE,
                 "%s: a 16-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    const size_t hi = (size_t)s * H * s * W;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float *region = static_cast<float *>(workspace) + (size_t)B * G * 25 * hi;      // the window weights (tensor type) live here
    OutlierTap *taps = reinterpret_cast<OutlierTap *>(region + (size_t)B * G * 25 * hi);
    unsigned int *tap_count = reinterpret_cast<unsigned int *>(taps + (size_t)B * G * hi);
    if (int e = clear_counter(fn, tap_count, st)) return e;
    // the attention is only read in this mode
    if (int e = SAPA_DISPATCH_FAST(dtype, [&] {
            launch_window<WIN_WEIGHTS, scalar_t>(P, B * G, hi, st, nullptr, nullptr, static_cast<const scalar_t *>(offset), nullptr,
                                                 const_cast<scalar_t *>(static_cast<const scalar_t *>(attn)), reinterpret_cast<scalar_t *>(region), taps, tap_count, B, C,
                                                 H, W, P, G, H, 0);
            return check_launch("deform_window_kernel<weights>");
        }))
        return e;
    if (int e = run_agg(region, value, out, B * G, C / G, H, W, 5, 2, dtype, st, G)) return e;
    return SAPA_DISPATCH_FAST(dtype, [&] {
        launch_next_with_l1(deform_outlier_kernel<scalar_t>, 148 * 8, 256, st, taps, tap_count, static_cast<const scalar_t *>(value),
                                                                 static_cast<const scalar_t *>(offset), static_cast<scalar_t *>(out), C, H,
                                                                 W, P, G, H, 0);
        return check_launch("deform_outlier_kernel");
    });
}

size_t sapa_deform_fused_backward_workspace(int B, int H, int W, int P, int s, int G, int dtype) {
    if (B <= 0 || H <= 0 || W <= 0 || P <= 0 || G <= 0 || s != 2) return 0;
    // 16-bit tensors: 16-bit operands in the tensor-core kernels, float32 similarities between them.  Rows that are not multiples of 16 bytes run the
    // float32 chain on widened tensors, or the gather kernels, with float32 weights
    if (dtype != SAPA_F32 && !((dtype == SAPA_F16 || dtype == SAPA_BF16) && fused_tma_supported(W, dtype))) return 0;
    const size_t hi = (size_t)s * H * s * W;
    if ((size_t)B * G * P >= 0xffffffffull || hi >= 0xffffffffull) return 0;
    // D, dWd (float32), dD, Wd (the tensors' type; sized for float32), the outlier list (worst case: every point) and
    // its counter
    return (size_t)B * G * 100 * hi * sizeof(float) + (size_t)B * G * P * hi * sizeof(OutlierGrad) + 16;
}

// 16-bit tensors only: float32 side buffers for the scattered key / value gradients of the listed points
size_t sapa_deform_fused_backward_scatter_bytes(int B, int Cq, int C, int H, int W, int dtype) {
    if (dtype != SAPA_F16 && dtype != SAPA_BF16) return 0;
    return ((size_t)B * Cq * H * W + (size_t)B * C * H * W) * sizeof(float);
}

int sapa_deform_fused_backward_dense(const void *grad_out, const void *query, const void *key, const void *value,
                                     const void *offset, const void *attn, void *grad_query, void *grad_key, void *grad_value,
                                     void *grad_offset, void *workspace, size_t workspace_bytes, int B, int Cq, int C, int H,
                                     int W, int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_fused_backward_dense";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, C, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, grad_out); SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, value);
    SAPA_CHECK_PTR(fn, offset); SAPA_CHECK_PTR(fn, attn); SAPA_CHECK_PTR(fn, grad_query); SAPA_CHECK_PTR(fn, grad_key);
    SAPA_CHECK_PTR(fn, grad_value); SAPA_CHECK_PTR(fn, grad_offset);
    const size_t base = sapa_deform_fused_backward_workspace(B, H, W, P, s, G, dtype);
    const size_t side_off = (base + 15) & ~(size_t)15;          // the side buffers of the 16-bit path start here
    const size_t need = side_off + sapa_deform_fused_backward_scatter_bytes(B, Cq, C, H, W, dtype);
    SAPA_REQUIRE(s == 2 && P <= MAXP && base != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: the dense-window path needs s = 2, num_point <= %d and float32, or float16 / bfloat16 with rows of 16 bytes "
                 "(use sapa_deform_fused_backward)", fn, MAXP);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && aligned16(workspace), SAPA_ERR_WORKSPACE,
                 "%s: a 16-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    const size_t hi = (size_t)s * H * s * W, plane = (size_t)B * G * 25 * hi;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // D and dWd are float32 whatever the tensors' type; dD and Wd are weights of the SAPA-B kernels and have the tensors'
    // type (those kernels round their weights to it anyway); every region is sized for float32
    float *dense = static_cast<float *>(workspace), *dwin = dense + plane;
    void *ddense = dwin + plane, *window = dwin + 2 * plane;
    OutlierGrad *taps = reinterpret_cast<OutlierGrad *>(dense + 4 * plane);
    unsigned int *tap_count = reinterpret_cast<unsigned int *>(taps + (size_t)B * G * P * hi);
    if (int e = clear_counter(fn, tap_count, st)) return e;
    // 1. D = sim(Q, Key) and dWd = sim(dOut, Value), the B x G groups as images
    if (dtype == SAPA_F32) {
        if (int e = run_sim(query, key, dense, B * G, Cq / G, H, W, 5, 2, dtype, st, G)) return e;
        if (int e = run_sim(grad_out, value, dwin, B * G, C / G, H, W, 5, 2, dtype, st, G)) return e;
    } else {
        if (int e = run_sim_mixed(query, key, dense, B * G, Cq / G, H, W, H, 0, dtype, st, G)) return e;
        if (int e = run_sim_mixed(grad_out, value, dwin, B * G, C / G, H, W, H, 0, dtype, st, G)) return e;
    }
    // 2. per pixel: softmax backward over the points, dD, Wd, offset gradients, list of the points outside the window
    {
        const int e = SAPA_DISPATCH_FAST(dtype, [&] {
            const scalar_t *go = static_cast<const scalar_t *>(grad_out), *v = static_cast<const scalar_t *>(value);
            const scalar_t *o = static_cast<const scalar_t *>(offset), *a = static_cast<const scalar_t *>(attn);
            scalar_t *dd = static_cast<scalar_t *>(ddense), *wn = static_cast<scalar_t *>(window), *goff = static_cast<scalar_t *>(grad_offset);
            launch_window_bwd<BWD_FUSED, scalar_t>(P, B * G, hi, st, go, v, o, a, static_cast<const float *>(dense), static_cast<const float *>(dwin), dd, wn, goff,
                                                   static_cast<scalar_t *>(nullptr), taps, tap_count, B, C, H, W, P, G);
            return check_launch("deform_window_bwd_kernel");
        });
        if (e) return e;
    }
    // 3. dQ = agg(dD, Key), dKey = gath(Q, dD), dV = gath(dOut, Wd): SAPA-B kernels per group, all outputs overwritten
    if (int e = run_agg(ddense, key, grad_query, B * G, Cq / G, H, W, 5, 2, dtype, st, G)) return e;
    if (int e = run_gath(query, ddense, grad_key, B * G, Cq / G, H, W, 5, 2, dtype, st, G)) return e;
    if (int e = run_gath(grad_out, window, grad_value, B * G, C / G, H, W, 5, 2, dtype, st, G)) return e;
    // 4. the listed points.  float32: atomics straight into the gradients.  16-bit: key / value contributions go to zeroed
    //    float32 side buffers behind the list and are folded into the 16-bit gradients by one more kernel.
    if (dtype == SAPA_F32) {
        launch_in_order(deform_outlier_bwd_kernel<float, float>, 148 * 8, 256, 0, st,
            taps, tap_count, static_cast<const float *>(grad_out), static_cast<const float *>(query), static_cast<const float *>(key),
            static_cast<const float *>(value), static_cast<const float *>(offset), static_cast<float *>(grad_query),
            static_cast<float *>(grad_key), static_cast<float *>(grad_value), static_cast<float *>(grad_offset), Cq, C, H, W, P, G);
        return check_launch("deform_outlier_bwd_kernel");
    }
    const size_t n_k = (size_t)B * Cq * H * W, n_v = (size_t)B * C * H * W;
    float *side_k = reinterpret_cast<float *>(static_cast<char *>(workspace) + side_off), *side_v = side_k + n_k;
    const Scatter sc{side_k, side_v, n_k, n_v, Cq / G, C / G};
    return SAPA_DISPATCH_FAST(dtype, [&] {
        launch_next(deform_zero_scatter_kernel<scalar_t>, 148 * 8, 256, 0, st, taps, tap_count, static_cast<const scalar_t *>(offset), sc, H, W, P);
        if (int e = check_launch("deform_zero_scatter_kernel")) return e;
        launch_in_order(deform_outlier_bwd_kernel<scalar_t, float>, 148 * 8, 256, 0, st,
            taps, tap_count, static_cast<const scalar_t *>(grad_out), static_cast<const scalar_t *>(query),
            static_cast<const scalar_t *>(key), static_cast<const scalar_t *>(value), static_cast<const scalar_t *>(offset),
            static_cast<scalar_t *>(grad_query), side_k, side_v, static_cast<scalar_t *>(grad_offset), Cq, C, H, W, P, G);
        if (int e = check_launch("deform_outlier_bwd_kernel")) return e;
        launch_next(deform_add_scatter_kernel<scalar_t>, 148 * 8, 256, 0, st, taps, tap_count, static_cast<const scalar_t *>(offset), sc, static_cast<scalar_t *>(grad_key),
                                                                     static_cast<scalar_t *>(grad_value), H, W, P);
        return check_launch("deform_add_scatter_kernel");
    });
}

// Backward of deform_av and of deform_qk alone through the dense window (s = 2, float32): the two halves of
// sapa_deform_fused_backward_dense without the softmax between them.  Workspace as for that entry point.
int sapa_deform_av_backward_dense(const void *grad_out, const void *attn, const void *value, const void *offset, void *grad_attn,
                                  void *grad_value, void *grad_offset, void *workspace, size_t workspace_bytes, int B, int C,
                                  int H, int W, int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_av_backward_dense";
    trace_reset();
    if (int e = check_deform(fn, B, C, C, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, grad_out); SAPA_CHECK_PTR(fn, attn); SAPA_CHECK_PTR(fn, value); SAPA_CHECK_PTR(fn, offset);
    SAPA_CHECK_PTR(fn, grad_attn); SAPA_CHECK_PTR(fn, grad_value); SAPA_CHECK_PTR(fn, grad_offset);
    const size_t base = sapa_deform_fused_backward_workspace(B, H, W, P, s, G, dtype);
    const size_t side_off = (base + 15) & ~(size_t)15;
    const size_t need = side_off + sapa_deform_fused_backward_scatter_bytes(B, 0, C, H, W, dtype);
    SAPA_REQUIRE(s == 2 && P <= MAXP && base != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: the dense-window path needs s = 2, num_point <= %d and float32, or float16 / bfloat16 with rows of 16 bytes "
                 "(use sapa_deform_av_backward)", fn, MAXP);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && aligned16(workspace), SAPA_ERR_WORKSPACE,
                 "%s: a 16-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    const size_t hi = (size_t)s * H * s * W, plane = (size_t)B * G * 25 * hi;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float *dwin = static_cast<float *>(workspace) + plane;
    void *window = dwin + 2 * plane;                                   // Wd, in the tensors' type
    OutlierGrad *taps = reinterpret_cast<OutlierGrad *>(static_cast<float *>(workspace) + 4 * plane);
    unsigned int *tap_count = reinterpret_cast<unsigned int *>(taps + (size_t)B * G * P * hi);
    if (int e = clear_counter(fn, tap_count, st)) return e;
    if (dtype == SAPA_F32) {
        if (int e = run_sim(grad_out, value, dwin, B * G, C / G, H, W, 5, 2, dtype, st, G)) return e;        // dWd
    } else {
        if (int e = run_sim_mixed(grad_out, value, dwin, B * G, C / G, H, W, H, 0, dtype, st, G)) return e;
    }
    if (int e = SAPA_DISPATCH_FAST(dtype, [&] {
            launch_window_bwd<BWD_AV, scalar_t>(P, B * G, hi, st, static_cast<const scalar_t *>(grad_out), static_cast<const scalar_t *>(value),
                                                static_cast<const scalar_t *>(offset), static_cast<const scalar_t *>(attn), static_cast<const float *>(nullptr),
                                                static_cast<const float *>(dwin), static_cast<scalar_t *>(nullptr), static_cast<scalar_t *>(window),
                                                static_cast<scalar_t *>(grad_offset), static_cast<scalar_t *>(grad_attn), taps, tap_count, B, C, H, W, P, G);
            return check_launch("deform_window_bwd_kernel<av>");
        }))
        return e;
    if (int e = run_gath(grad_out, window, grad_value, B * G, C / G, H, W, 5, 2, dtype, st, G)) return e;  // dV
    if (dtype == SAPA_F32) {
        launch_in_order(deform_outlier_bwd_kernel<float, float>, 148 * 8, 256, 0, st,
            taps, tap_count, static_cast<const float *>(grad_out), nullptr, nullptr, static_cast<const float *>(value),
            static_cast<const float *>(offset), nullptr, nullptr, static_cast<float *>(grad_value), static_cast<float *>(grad_offset),
            C, C, H, W, P, G);
        return check_launch("deform_outlier_bwd_kernel");
    }
    const size_t n_v = (size_t)B * C * H * W;
    float *side_v = reinterpret_cast<float *>(static_cast<char *>(workspace) + side_off);
    const Scatter sc{nullptr, side_v, 0, n_v, 0, C / G};
    return SAPA_DISPATCH_FAST(dtype, [&] {
        launch_next(deform_zero_scatter_kernel<scalar_t>, 148 * 8, 256, 0, st, taps, tap_count, static_cast<const scalar_t *>(offset), sc, H, W, P);
        if (int e = check_launch("deform_zero_scatter_kernel")) return e;
        launch_in_order(deform_outlier_bwd_kernel<scalar_t, float>, 148 * 8, 256, 0, st,
            taps, tap_count, static_cast<const scalar_t *>(grad_out), nullptr, nullptr, static_cast<const scalar_t *>(value),
            static_cast<const scalar_t *>(offset), nullptr, nullptr, side_v, static_cast<scalar_t *>(grad_offset), C, C, H, W, P, G);
        if (int e = check_launch("deform_outlier_bwd_kernel")) return e;
        launch_next(deform_add_scatter_kernel<scalar_t>, 148 * 8, 256, 0, st, taps, tap_count, static_cast<const scalar_t *>(offset), sc, static_cast<scalar_t *>(nullptr),
                                                                     static_cast<scalar_t *>(grad_value), H, W, P);
        return check_launch("deform_add_scatter_kernel");
    });
}

int sapa_deform_qk_backward_dense(const void *grad_out, const void *query, const void *key, const void *offset, void *grad_query,
                                  void *grad_key, void *grad_offset, void *workspace, size_t workspace_bytes, int B, int Cq,
                                  int H, int W, int P, int s, int G, int dtype, void *stream) {
    const char *fn = "sapa_deform_qk_backward_dense";
    trace_reset();
    if (int e = check_deform(fn, B, Cq, Cq, H, W, P, s, G, dtype)) return e;
    SAPA_CHECK_PTR(fn, grad_out); SAPA_CHECK_PTR(fn, query); SAPA_CHECK_PTR(fn, key); SAPA_CHECK_PTR(fn, offset);
    SAPA_CHECK_PTR(fn, grad_query); SAPA_CHECK_PTR(fn, grad_key); SAPA_CHECK_PTR(fn, grad_offset);
    const size_t base = sapa_deform_fused_backward_workspace(B, H, W, P, s, G, dtype);
    const size_t side_off = (base + 15) & ~(size_t)15;
    const size_t need = side_off + sapa_deform_fused_backward_scatter_bytes(B, Cq, 0, H, W, dtype);
    SAPA_REQUIRE(s == 2 && P <= MAXP && base != 0, SAPA_ERR_UNSUPPORTED,
                 "%s: the dense-window path needs s = 2, num_point <= %d and float32, or float16 / bfloat16 with rows of 16 bytes "
                 "(use sapa_deform_qk_backward)", fn, MAXP);
    SAPA_REQUIRE(workspace != nullptr && workspace_bytes >= need && aligned16(workspace), SAPA_ERR_WORKSPACE,
                 "%s: a 16-byte aligned workspace of %zu bytes is required, got %zu", fn, need, workspace_bytes);
    const size_t hi = (size_t)s * H * s * W, plane = (size_t)B * G * 25 * hi;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float *dense = static_cast<float *>(workspace);
    void *ddense = dense + 2 * plane;                                  // dD, in the tensors' type
    OutlierGrad *taps = reinterpret_cast<OutlierGrad *>(dense + 4 * plane);
    unsigned int *tap_count = reinterpret_cast<unsigned int *>(taps + (size_t)B * G * P * hi);
    if (int e = clear_counter(fn, tap_count, st)) return e;
    if (dtype == SAPA_F32) {
        if (int e = run_sim(query, key, dense, B * G, Cq / G, H, W, 5, 2, dtype, st, G)) return e;         // D, for the offset gradients
    } else {
        if (int e = run_sim_mixed(query, key, dense, B * G, Cq / G, H, W, H, 0, dtype, st, G)) return e;
    }
    // the logit gradients enter where the fused chain reads the attention
    if (int e = SAPA_DISPATCH_FAST(dtype, [&] {
            launch_window_bwd<BWD_QK, scalar_t>(P, B * G, hi, st, static_cast<const scalar_t *>(nullptr), static_cast<const scalar_t *>(nullptr),
                                                static_cast<const scalar_t *>(offset), static_cast<const scalar_t *>(grad_out), static_cast<const float *>(dense),
                                                static_cast<const float *>(nullptr), static_cast<scalar_t *>(ddense), static_cast<scalar_t *>(nullptr),
                                                static_cast<scalar_t *>(grad_offset), static_cast<scalar_t *>(nullptr), taps, tap_count, B, Cq, H, W, P, G);
            return check_launch("deform_window_bwd_kernel<qk>");
        }))
        return e;
    if (int e = run_agg(ddense, key, grad_query, B * G, Cq / G, H, W, 5, 2, dtype, st, G)) return e;       // dQ
    if (int e = run_gath(query, ddense, grad_key, B * G, Cq / G, H, W, 5, 2, dtype, st, G)) return e;      // dKey
    if (dtype == SAPA_F32) {
        launch_in_order(deform_outlier_bwd_kernel<float, float>, 148 * 8, 256, 0, st,
            taps, tap_count, nullptr, static_cast<const float *>(query), static_cast<const float *>(key), nullptr,
            static_cast<const float *>(offset), static_cast<float *>(grad_query), static_cast<float *>(grad_key), nullptr,
            static_cast<float *>(grad_offset), Cq, Cq, H, W, P, G);
        return check_launch("deform_outlier_bwd_kernel");
    }
    const size_t n_k = (size_t)B * Cq * H * W;
    float *side_k = reinterpret_cast<float *>(static_cast<char *>(workspace) + side_off);
    const Scatter sc{side_k, nullptr, n_k, 0, Cq / G, 0};
    return SAPA_DISPATCH_FAST(dtype, [&] {
        launch_next(deform_zero_scatter_kernel<scalar_t>, 148 * 8, 256, 0, st, taps, tap_count, static_cast<const scalar_t *>(offset), sc, H, W, P);
        if (int e = check_launch("deform_zero_scatter_kernel")) return e;
        launch_in_order(deform_outlier_bwd_kernel<scalar_t, float>, 148 * 8, 256, 0, st,
            taps, tap_count, nullptr, static_cast<const scalar_t *>(query), static_cast<const scalar_t *>(key), nullptr,
            static_cast<const scalar_t *>(offset), static_cast<scalar_t *>(grad_query), side_k, nullptr,
            static_cast<scalar_t *>(grad_offset), Cq, Cq, H, W, P, G);
        if (int e = check_launch("deform_outlier_bwd_kernel")) return e;
        launch_next(deform_add_scatter_kernel<scalar_t>, 148 * 8, 256, 0, st, taps, tap_count, static_cast<const scalar_t *>(offset), sc, static_cast<scalar_t *>(grad_key),
                                                                     static_cast<scalar_t *>(nullptr), H, W, P);
        return check_launch("deform_add_scatter_kernel");
    });
}

}  // extern "C"
