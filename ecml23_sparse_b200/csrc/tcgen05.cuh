// Thin wrappers of the fifth-generation tensor core instructions (tcgen05, TMEM, mbarrier): for the forward that densifies tiles
// of the weight table (forward_dense.cu), and for the one-pass backward, which keeps sums and inputs in tensor memory
// (backward_fused.cu).  The MMA has one form here:
//   D[128][n] (+)= A[128][16] * B[n][16]^T,  bf16 operands, fp32 accumulation,
// A and D in tensor memory, B in shared memory, K-major in panels of 64 elements (128 bytes) with the 128-byte swizzle.
#pragma once

#include "ffi_common.cuh"

namespace ffi {
namespace tc {

constexpr int kCols = 512;       // TMEM columns of an SM; these kernels run one CTA per SM and take them all
constexpr int kPanelK = 64;      // elements of K per shared-memory panel (one 128-byte row)

__device__ __forceinline__ unsigned smem_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void alloc(void* smem_dst) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(smem_dst)), "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void dealloc(unsigned base) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(kCols) : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Orders this thread's generic-proxy accesses to shared memory before later reads of the tensor core or copies of the TMA unit.
__device__ __forceinline__ void fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 8 consecutive columns of this thread's TMEM lane
__device__ __forceinline__ void store8(unsigned taddr, const unsigned (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// 16 consecutive columns, complete on return
__device__ __forceinline__ void load16(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}
// One column each, at base + c0 ... base + c3, complete on return
__device__ __forceinline__ void load_columns(unsigned base, unsigned c0, unsigned c1, unsigned c2, unsigned c3, unsigned (&r)[4]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%4];\n"
        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%1}, [%5];\n"
        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%2}, [%6];\n"
        "tcgen05.ld.sync.aligned.32x32b.x1.b32 {%3}, [%7];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3])
        : "r"(base + c0), "r"(base + c1), "r"(base + c2), "r"(base + c3)
        : "memory");
}

// Shared-memory descriptor of a K-major panel with the 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes
// apart; the panel starts on a 1024-byte boundary and K advances by 32 bytes per MMA inside a row.
__device__ __forceinline__ unsigned long long panel_desc(unsigned addr) {
    return static_cast<unsigned long long>((addr & 0x3ffffu) >> 4) | (1ull << 16) | (static_cast<unsigned long long>(1024 >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// The descriptor of what lies `bytes` (a multiple of 16) behind it
__device__ __forceinline__ unsigned long long desc_at(unsigned long long desc, unsigned bytes) { return desc + (bytes >> 4); }
// Byte offset of element (row, k) of a panel, k < 64.
__device__ __forceinline__ unsigned panel_offset(unsigned row, unsigned k) { return row * 128u + ((2u * k) ^ ((row & 7u) << 4)); }

// Instruction descriptor: fp32 D, bf16 A and B, both K-major, M = 128.
__host__ __device__ constexpr unsigned instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<unsigned>(n >> 3) << 17) | (static_cast<unsigned>(128 >> 4) << 24);
}
__device__ __forceinline__ void mma(unsigned d, unsigned a, unsigned long long b_desc, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d),
        "r"(a), "l"(b_desc), "r"(idesc), "r"(static_cast<unsigned>(accumulate))
        : "memory");
}
// All MMAs this thread issued before arrive on `bar` when they are done.
__device__ __forceinline__ void commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void bar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool bar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Waits for the phase with the given parity, at most `limit` clock64 ticks; false if it gave up.
__device__ __forceinline__ bool bar_wait(unsigned long long* bar, unsigned parity, long long limit) {
    if (bar_try_wait(bar, parity)) return true;
    const long long start = clock64();
    while (!bar_try_wait(bar, parity))
        if (clock64() - start > limit) return false;
    return true;
}

}  // namespace tc
}  // namespace ffi
