// tcgen05 kind::i8 building blocks for kernels that put exact integer contractions on the tensor cores: unsigned bytes of
// 64-bit words, 32-bit sums in tensor memory. Operands live in shared memory in the 128-byte swizzle (rows of 128 bytes,
// the 16-byte unit u of row r at u ^ (r mod 8), groups of eight rows 1024 bytes apart), which 16-byte stores of a warp
// and 16-byte asynchronous copies write without bank conflicts:
//   K-major    row = row of M or N, its 128 bytes = K; the next 32 of K are 32 bytes on;
//   MN-major   row = index of K, its 128 bytes = M or N; the next 32 of K are 32 rows (4096 bytes) on; a second 128 of N
//              lies `lead` bytes on.
// Waits are bounded. Where one runs out a kernel goes on to its end without waiting again, so that every barrier is met; the thread that
// issues MMAs waits (Issued::drain) for those in flight before tensor memory is freed. A kernel whose results are a block's own
// then forms them again from memory (rows of a partial evaluation, hashes). One whose results are sums over all blocks cannot: it sets
// an error word for the host, which fails the proof and discards the scratch.
// Measured: an MMA of M = 128, K = 32 takes the pipe 59 cycles up to N = 64, 64 at N = 128, 128 at N = 256, whichever
// layout its operands have.
#pragma once
#include <stdint.h>

namespace mb {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// byte offset of 16-byte unit u of row r
__device__ __forceinline__ uint32_t swz(uint32_t r, uint32_t u) { return r * 128 + ((u ^ (r & 7)) << 4); }

__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr, uint32_t lead) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lead >> 4) & 0x3FFF) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ULL << 46) |
           (2ULL << 61);
}
// D = s32, A = B = u8, M = 128
__host__ __device__ constexpr uint32_t idesc_u8(int n, bool mn_major) {
    return (2u << 4) | (mn_major ? 3u << 15 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
// the mbarrier completes once every MMA this thread has issued is done
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// shared memory written by this thread (stores, finished asynchronous copies) is visible to the MMAs issued after a barrier
__device__ __forceinline__ void fence_operands() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// a warp's call; cols a power of two from 32
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// barrier of `threads` threads of a block, id from 1
__device__ __forceinline__ void named_sync(uint32_t threads, uint32_t id = 1) { asm volatile("bar.sync %1, %0;" ::"r"(threads), "r"(id) : "memory"); }
// all threads of the cluster: what they wrote to shared memory is there for the others
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// bounded: false after `polls` polls. MB_TC_POLLS: 0 in a test build, where every wait of a kernel but Issued::drain runs out at once.
#ifndef MB_TC_POLLS
#define MB_TC_POLLS (1 << 20)
#endif
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int polls = MB_TC_POLLS) {
    for (int it = 0; it < polls; it++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// What a thread has issued: the last barrier that it committed its MMAs to. drain: every MMA before that is done, or a million polls are.
struct Issued {
    uint32_t bar = ~0u, parity = 0;
    __device__ __forceinline__ void commit_to(uint32_t b, uint32_t phase) {
        commit(b);
        bar = b;
        parity = phase & 1;
    }
    __device__ __forceinline__ void drain() const {
        if (bar != ~0u) mbar_wait(bar, parity, 1 << 20);
    }
};
// eight or sixteen columns from addr of the calling thread's lane; complete on return
__device__ __forceinline__ void ld8(uint32_t addr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ld16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                   "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(addr) : "memory");
}
// 16 bytes to shared memory, asynchronously, past L1
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

}  // namespace tc
}  // namespace mb
