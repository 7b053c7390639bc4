// finite.cuh — infinities and NaN in front of a banded product.  The kernels on strips multiply a landed row of one operand with weights that
// are zero outside a pixel's window, and 0 * inf would reach outputs that no infinity reaches.  So the warps that move a row into tensor
// memory move zeros in place of what is not finite and note the row; when a CTA has stored all its outputs, it looks at the elements of the noted
// rows in memory and stores again the outputs whose windows hold one that is not finite, as what they come to.  Rows are checked with an FMA for
// one or two elements while they are on their way; nothing else is done while all numbers are finite.  (Outputs put right in front of their store
// cost registers in every step: 8 x 256 x 64x64 forward in bfloat16 27.0 -> 29.1 us.)
#pragma once

#include "tma_util.cuh"

namespace sapa {
namespace finite {

// whether all elements of N words are finite: x * 0 summed is zero then, NaN else
template <typename T, int N> __device__ __forceinline__ bool all_finite(const unsigned *v) {
    if constexpr (sizeof(T) == 4) {
        float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < N; ++i) z[i & 3] = fmaf(__uint_as_float(v[i]), 0.f, z[i & 3]);
        return (z[0] + z[1]) + (z[2] + z[3]) == 0.f;
    } else {
        using P = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
        unsigned z[4] = {0u, 0u, 0u, 0u};
        const unsigned zero = 0u;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const P s = __hfma2(*reinterpret_cast<const P *>(&v[i]), *reinterpret_cast<const P *>(&zero), *reinterpret_cast<const P *>(&z[i & 3]));
            z[i & 3] = *reinterpret_cast<const unsigned *>(&s);
        }
        return ((z[0] | z[1] | z[2] | z[3]) & 0x7fff7fffu) == 0u;      // a zero of either sign
    }
}
// the bits of an element's exponent
template <typename T> __device__ __forceinline__ constexpr unsigned exponent() { return sizeof(T) == 4 ? 0x7f800000u : std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u; }
// one of four registers, at a place known at run time
__device__ __forceinline__ unsigned pick(const unsigned (&v)[4], int i) { return i < 2 ? (i == 0 ? v[0] : v[1]) : i == 2 ? v[2] : v[3]; }
// element e of 16 bytes
template <typename T> __device__ __forceinline__ bool is_finite(const unsigned (&v)[4], int e) {
    const unsigned u = sizeof(T) == 4 ? pick(v, e) : pick(v, e >> 1) >> (e & 1) * 16;
    return (u & exponent<T>()) != exponent<T>();
}
// a word with zeros in place of its elements that are not finite
template <typename T> __device__ __forceinline__ unsigned or_zero(unsigned u) {
    if constexpr (sizeof(T) == 4) {
        return (u & 0x7f800000u) == 0x7f800000u ? 0u : u;
    } else {
        constexpr unsigned E = exponent<T>(), EXP = E | E << 16, ONE = E & (0u - E);      // the exponent's lowest bit
        const unsigned odd = ((u & EXP) + (ONE | ONE << 16)) & 0x80008000u;      // an exponent of ones runs over into the sign's place, no further
        return u & ~((odd >> 15) * 0xffffu);
    }
}

// Columns of a row that hold NaN, +inf, -inf: bit i = column from + i (PAIRS: columns from + 2i and from + 2i + 1), of VECS chunks of 16 bytes, each wholly
// inside the row's W columns or outside.
struct Marks {
    unsigned long long nan, up, down;
    __device__ __forceinline__ unsigned long long any() const { return nan | up | down; }
};
template <typename T, int VECS, bool PAIRS>
__device__ __noinline__ void mark_row(const T *row, int W, int from, Marks &m) {
    constexpr int PER = 16 / (int)sizeof(T);
    uint4 w[VECS];
#pragma unroll
    for (int j = 0; j < VECS; ++j) {
        const int x = from + j * PER;
        w[j] = x >= 0 && x < W ? *reinterpret_cast<const uint4 *>(row + x) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int j = 0; j < VECS; ++j) {
        const unsigned words[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
        if (all_finite<T, 4>(words)) continue;
#pragma unroll 1
        for (int e = 0; e < PER; ++e) {
            const unsigned u = sizeof(T) == 4 ? pick(words, e) : pick(words, e >> 1) >> (e & 1) * 16 << 16;      // the element in the high bits
            constexpr unsigned SIGN = 0x80000000u, TOP = exponent<T>() << (sizeof(T) == 4 ? 0 : 16);
            const unsigned long long bit = 1ull << ((j * PER + e) >> (PAIRS ? 1 : 0));
            if ((u & ~SIGN) > TOP) m.nan |= bit;
            else if (u == TOP) m.up |= bit;
            else if (u == (TOP | SIGN)) m.down |= bit;
        }
    }
}
// First and last noted row (in the order in which a CTA takes them) of the 32 channels of a warp; whether one was for a sum that is not finite
struct Noted {
    int first[4], last[4], sums[4];
    __device__ __forceinline__ void clear(int i) { first[i] = 0x7fffffff; last[i] = -1; sums[i] = 0; }
    __device__ __forceinline__ void note(int quarter, int row) { atomicMin(&first[quarter], row); atomicMax(&last[quarter], row); }
    __device__ __forceinline__ void note_sum(int quarter, int row) { note(quarter, row); sums[quarter] = 1; }
};
// whether 16 bytes hold nothing but NaN
template <typename T> __device__ __forceinline__ bool all_nan(const uint4 w) {
    const unsigned v[4] = {w.x, w.y, w.z, w.w};
    bool nan = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (sizeof(T) == 4) nan = nan && (v[i] & 0x7fffffffu) > exponent<T>();
        else nan = nan && (v[i] & 0x7fffu) > exponent<T>() && (v[i] >> 16 & 0x7fffu) > exponent<T>();
    }
    return nan;
}
// element e of 16 bytes as float32
template <typename T> __device__ __forceinline__ float element(const uint4 w, int e) {
    const unsigned v[4] = {w.x, w.y, w.z, w.w};
    if constexpr (sizeof(T) == 4) {
        return __uint_as_float(v[e]);
    } else {
        const float2 f = tmau::unpack_pair(T(), v[e >> 1]);
        return e & 1 ? f.y : f.x;
    }
}
// 16 bytes of NaN
template <typename T> __device__ __forceinline__ uint4 nan_chunk() {
    const unsigned u = sizeof(T) == 4 ? 0x7fffffffu : 0x7fff7fffu;
    return make_uint4(u, u, u, u);
}
__device__ __forceinline__ float nan_value() { return __int_as_float(0x7fffffff); }

}  // namespace finite
}  // namespace sapa
