// umma_util.cuh — PTX wrappers of the 5th-generation tensor core (tcgen05 and tensor memory) shared by the kernels that use it.
#pragma once

#include "tma_util.cuh"

namespace sapa {
namespace ummau {

using namespace tmau;

__device__ __forceinline__ void tc_alloc(unsigned smem_slot, unsigned ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_slot), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(unsigned taddr, unsigned ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// Bounded wait of a whole warp, in front of instructions that all of its lanes execute together: every lane gets the same answer.
__device__ __forceinline__ bool mbar_wait_warp(unsigned bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity)); }
// One tcgen05.mma, for a loop that the WHOLE warp runs with values the compiler can see to be the same in all lanes (warp index and
// addresses through warp_uniform): the operands stay in uniform registers, the lane with `leader` issues.  Measured (M = 128, tf32 and
// bf16): N / 2 clocks an instruction and 16 at least; in a branch that one lane takes, where every operand is moved to a uniform register
// first, 57 at least.  Shared-memory descriptors are passed as their low words (start address and leading offset; the part that changes from
// instruction to instruction) plus the high word that a kernel's operands share.
template <bool TF32>
__device__ __forceinline__ void tc_mma(unsigned leader, unsigned d_tmem, unsigned a_lo, unsigned b_lo, unsigned desc_hi, unsigned idesc, unsigned accumulate) {
    if (TF32)
        asm volatile("{\n .reg .pred p, q;\n .reg .b64 da, db;\n setp.ne.b32 p, %5, 0;\n setp.ne.b32 q, %6, 0;\n mov.b64 da, {%1, %3};\n mov.b64 db, {%2, %3};\n"
                     " @q tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %4, p;\n}\n"
                     ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
    else
        asm volatile("{\n .reg .pred p, q;\n .reg .b64 da, db;\n setp.ne.b32 p, %5, 0;\n setp.ne.b32 q, %6, 0;\n mov.b64 da, {%1, %3};\n mov.b64 db, {%2, %3};\n"
                     " @q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n}\n"
                     ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// The same with the A operand in tensor memory: lane = row of A, column = 32 bits of its K dimension (one tf32 or two 16-bit elements).
template <bool TF32>
__device__ __forceinline__ void tc_mma_ta(unsigned leader, unsigned d_tmem, unsigned a_tmem, unsigned b_lo, unsigned desc_hi, unsigned idesc, unsigned accumulate) {
    if (TF32)
        asm volatile("{\n .reg .pred p, q;\n .reg .b64 db;\n setp.ne.b32 p, %5, 0;\n setp.ne.b32 q, %6, 0;\n mov.b64 db, {%2, %3};\n"
                     " @q tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], db, %4, p;\n}\n"
                     ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
    else
        asm volatile("{\n .reg .pred p, q;\n .reg .b64 db;\n setp.ne.b32 p, %5, 0;\n setp.ne.b32 q, %6, 0;\n mov.b64 db, {%2, %3};\n"
                     " @q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n}\n"
                     ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// the mbarrier receives one arrival when every tcgen05.mma that the leader has issued so far has completed
__device__ __forceinline__ void tc_commit_by(unsigned leader, unsigned bar) {
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n"
                 ::"r"(bar), "r"(leader) : "memory");
}
// 1 in one lane of a converged warp
__device__ __forceinline__ unsigned elect_leader() {
    unsigned leader;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(leader));
    return leader;
}
__device__ __forceinline__ unsigned warp_uniform(unsigned v) { return __shfl_sync(0xffffffffu, v, 0); }
// 16 consecutive accumulator columns of this thread's lane
__device__ __forceinline__ void tc_ld16(unsigned taddr, unsigned (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// 8 and 16 consecutive columns of this thread's lane, from registers
__device__ __forceinline__ void tc_st8(unsigned taddr, const unsigned *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};\n"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_st16(unsigned taddr, const unsigned *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};\n"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// low word of a shared-memory matrix descriptor: start address (bits 0-13) and leading byte offset (bits 16-29) in 16-byte units
__device__ __forceinline__ unsigned desc_lo(unsigned addr, unsigned leading_bytes) {
    return ((addr & 0x3ffffu) >> 4) | ((leading_bytes >> 4) << 16);
}

template <typename T> struct UmmaFormat;
template <> struct UmmaFormat<float> { static constexpr unsigned code = 2; };            // tf32
template <> struct UmmaFormat<__half> { static constexpr unsigned code = 0; };
template <> struct UmmaFormat<__nv_bfloat16> { static constexpr unsigned code = 1; };

// instruction descriptor but for N: float32 accumulator, both operands T, K-major, M = 128
template <typename T> constexpr unsigned IDESC_M128 = (1u << 4) | (UmmaFormat<T>::code << 7) | (UmmaFormat<T>::code << 10) | ((128u >> 4) << 24);
__device__ __forceinline__ constexpr unsigned idesc_n(unsigned n) { return (n >> 3) << 17; }

// ---------------------------------------------------------------------------------- host side
// Kernels that walk `columns` (strips of all images and blocks of channels) of `rows` rows each: cuts every column into `segs` items of
// `seg_rows` rows so that the busiest of the SMs takes the fewest steps, an item costing `extra` steps beyond its rows and the launch three.
// The candidates are the most segments that one, two, ... rounds of items hold.
inline void split_rows(long long columns, int rows, int sms, int extra, long long &items, long long &steps, int &seg_rows, int &segs) {
    const int first = (int)((columns + sms - 1) / sms);
    items = 0;
    for (int round = first; round < first + 5; ++round) {
        const long long most = (long long)round * sms / columns;
        const int want = most < rows ? (int)most : rows, r = (rows + want - 1) / want, used = (rows + r - 1) / r;
        const long long n = columns * used, total = (n + sms - 1) / sms * (r + extra) + 3;
        if (items != 0 && total >= steps) continue;
        items = n; steps = total; seg_rows = r; segs = used;
    }
}

}  // namespace ummau
}  // namespace sapa
