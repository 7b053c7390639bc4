// common.cuh — element-type traits, small device helpers and host-side error plumbing shared by the
// SAPA kernels.  Everything computes in an accumulation type (float for f32/f16/bf16, double for f64).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "../../include/sapa_b200.h"

namespace sapa {

// ---------------------------------------------------------------------------------- type traits
template <typename T> struct AccOf { using type = float; };
template <> struct AccOf<double> { using type = double; };

__device__ __forceinline__ float to_acc(float x) { return x; }
__device__ __forceinline__ float to_acc(__half x) { return __half2float(x); }
__device__ __forceinline__ float to_acc(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ double to_acc(double x) { return x; }

template <typename T> __device__ __forceinline__ T from_acc(typename AccOf<T>::type x);
template <> __device__ __forceinline__ float from_acc<float>(float x) { return x; }
template <> __device__ __forceinline__ __half from_acc<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_acc<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ double from_acc<double>(double x) { return x; }

// Streaming (evict-first) load / store of two adjacent elements (the two high-res columns of one low-res
// parent when s == 2) as one 64-bit or 32-bit access.  The 16-bit types go through `unsigned int` builtins:
// the toolkit's own __stcs overloads for __half2 / __nv_bfloat162 are inline asm with a "memory" clobber,
// which pins every shared-memory load behind the previous store and serialises the aggregation loop.
template <typename T> __device__ __forceinline__ float2 load_pair(const T *p);
template <> __device__ __forceinline__ float2 load_pair<float>(const float *p) {
    return __ldcs(reinterpret_cast<const float2 *>(p));
}
template <> __device__ __forceinline__ float2 load_pair<__half>(const __half *p) {
    const unsigned int raw = __ldcs(reinterpret_cast<const unsigned int *>(p));
    return __half22float2(*reinterpret_cast<const __half2 *>(&raw));
}
template <> __device__ __forceinline__ float2 load_pair<__nv_bfloat16>(const __nv_bfloat16 *p) {
    const unsigned int raw = __ldcs(reinterpret_cast<const unsigned int *>(p));
    return make_float2(__uint_as_float(raw << 16), __uint_as_float(raw & 0xffff0000u));
}

template <typename T> __device__ __forceinline__ void store_pair(T *p, float a, float b);
template <> __device__ __forceinline__ void store_pair<float>(float *p, float a, float b) {
    __stcs(reinterpret_cast<float2 *>(p), make_float2(a, b));
}
template <> __device__ __forceinline__ void store_pair<__half>(__half *p, float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    __stcs(reinterpret_cast<unsigned int *>(p), *reinterpret_cast<const unsigned int *>(&h));
}
template <> __device__ __forceinline__ void store_pair<__nv_bfloat16>(__nv_bfloat16 *p, float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    __stcs(reinterpret_cast<unsigned int *>(p), *reinterpret_cast<const unsigned int *>(&h));
}

// First thing in a kernel that is launched with launch_next, before any access to global memory: waits until the previous kernel of
// the stream has finished and its writes are visible, then lets the blocks of the next one be set up as this kernel's leave room.
// Such a kernel is alive while the previous one still writes what it will read, so nothing that it reads is "read-only for the
// lifetime of the kernel": no __ldg, and no pointer that it reads through is __restrict__ (the compiler makes the same load of a const
// one, and may move either ahead of the wait).  Plain loads, load_current and __ldcs stay behind it.
__device__ __forceinline__ void begin_after_previous() {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// A volatile load through the coherent path (the toolkit's 16-bit __ldca is not volatile, so those types go as unsigned short), for the
// kernels in which a plain load is slower: forward with K = 3, 8 x 128 x 64x64, float32 34.8 us with plain loads, 32.4 with these;
// bfloat16 58.8 and 46.4.
template <typename T> __device__ __forceinline__ T load_current(const T *p) {
    if constexpr (sizeof(T) == 2) {
        const unsigned short raw = __ldca(reinterpret_cast<const unsigned short *>(p));
        return *reinterpret_cast<const T *>(&raw);
    } else {
        return __ldca(p);
    }
}

__device__ __forceinline__ void atomic_add(float *p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add(double *p, double v) { atomicAdd(p, v); }

// ---------------------------------------------------------------------------------- host helpers
void set_error(const char *fmt, ...);   // stores a thread-local message, see api.cu
int check_launch(const char *what);     // cudaGetLastError() -> SAPA_OK (and records `what`) / SAPA_ERR_LAUNCH
void trace_reset();                     // start of an entry point: forget the kernels of the previous call
void trace_kernel(const char *name);    // appended by check_launch: read back through sapa_last_kernels()

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

inline size_t dtype_size(int dtype) {
    switch (dtype) {
        case SAPA_F32: return 4;
        case SAPA_F16: return 2;
        case SAPA_BF16: return 2;
        case SAPA_F64: return 8;
        default: return 0;
    }
}

inline int ceil_div(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }

#define SAPA_REQUIRE(cond, code, ...)      \
    do {                                   \
        if (!(cond)) {                     \
            ::sapa::set_error(__VA_ARGS__); \
            return (code);                 \
        }                                  \
    } while (0)

// every tensor pointer must be non-null and aligned to its element size; 16-byte alignment is only needed by the
// vectorised / tiled / tensor-map kernels and is checked where those are chosen (all_aligned16)
// (uses the entry point's `dtype` argument)
#define SAPA_CHECK_PTR(fn, p)                                                                                  \
    do {                                                                                                       \
        SAPA_REQUIRE((p) != nullptr, SAPA_ERR_ARGUMENT, "%s: %s is NULL", fn, #p);                              \
        SAPA_REQUIRE(::sapa::dtype_size(dtype) != 0 && reinterpret_cast<uintptr_t>(p) % ::sapa::dtype_size(dtype) == 0, \
                     SAPA_ERR_ALIGNMENT, "%s: %s is not aligned to the element size", fn, #p);                  \
    } while (0)

template <typename... P> inline bool all_aligned16(const P *...p) { return (aligned16(p) && ...); }

// Launch of a kernel that starts with begin_after_previous(): its blocks may be set up while the previous kernel of the stream drains
// (programmatic dependent launch), which hides the launch latency between the kernels of a chain, about 1.5 us of 2.5: three
// chained SAPA modules (twelve kernels) 253.6 -> 231.5 us, one SAPADeform module (six) 57.4 -> 50.3.
template <typename... P, typename... A>
inline void launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute attribute;
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid; config.blockDim = block; config.dynamicSmemBytes = smem; config.stream = st;
    config.attrs = &attribute; config.numAttrs = 1;
    (void)cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);      // a failure is what check_launch reads
}

// Kernels that live on the L1 cache (gathers, neighbours' overlapping reads).  An SM divides its memory between L1 and shared memory when
// it is empty: blocks set up beside a kernel with 200 KB of shared memory keep what that one left them.  So such a kernel is launched
// after the previous one has ended; or ahead with all of the memory asked for as L1, which holds it back from an SM until that is empty
// and is right only for a kernel without shared memory.  SAPA-D with sigma 1.5 (8 x 256 x 64x64, float32), its list kernels: launched as
// above 2037 (forward) and 3270 us (backward), in order 1207 and 2820, ahead with L1 1211 and 3068; its backward window kernel 950 as
// above, 838 in order.
template <typename... P, typename... A>
inline void launch_in_order(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    kernel<<<grid, block, smem, st>>>(static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline void launch_next_with_l1(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    attribute[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attribute[1].val.sharedMemCarveout = cudaSharedmemCarveoutMaxL1;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid; config.blockDim = block; config.stream = st;
    config.attrs = attribute; config.numAttrs = 2;
    (void)cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
}

// Runs the lambda body with `scalar_t` bound to the element type named by the dtype code.
// SAPA_DISPATCH_FAST: f32 / f16 / bf16 (tiled kernels).  SAPA_DISPATCH_ALL adds f64 (generic kernels).
#define SAPA_DISPATCH_CASE_(code, type, ...) \
    case code: {                             \
        using scalar_t = type;               \
        return __VA_ARGS__();                \
    }
#define SAPA_DISPATCH_FAST(dtype, ...)                                           \
    [&]() -> int {                                                               \
        switch (dtype) {                                                         \
            SAPA_DISPATCH_CASE_(SAPA_F32, float, __VA_ARGS__)                    \
            SAPA_DISPATCH_CASE_(SAPA_F16, __half, __VA_ARGS__)                   \
            SAPA_DISPATCH_CASE_(SAPA_BF16, __nv_bfloat16, __VA_ARGS__)           \
            default:                                                             \
                ::sapa::set_error("dtype code %d has no tiled kernel", (int)(dtype)); \
                return SAPA_ERR_DTYPE;                                           \
        }                                                                        \
    }()
#define SAPA_DISPATCH_ALL(dtype, ...)                                            \
    [&]() -> int {                                                               \
        switch (dtype) {                                                         \
            SAPA_DISPATCH_CASE_(SAPA_F32, float, __VA_ARGS__)                    \
            SAPA_DISPATCH_CASE_(SAPA_F16, __half, __VA_ARGS__)                   \
            SAPA_DISPATCH_CASE_(SAPA_BF16, __nv_bfloat16, __VA_ARGS__)           \
            SAPA_DISPATCH_CASE_(SAPA_F64, double, __VA_ARGS__)                   \
            default:                                                             \
                ::sapa::set_error("unknown dtype code %d", (int)(dtype));        \
                return SAPA_ERR_DTYPE;                                           \
        }                                                                        \
    }()

}  // namespace sapa
