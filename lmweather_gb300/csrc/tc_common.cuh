// tcgen05 / bulk-copy / mbarrier helpers for sm_103a kernels whose operands sit in global memory already in the
// MMA's canonical K-major core-matrix order (8 rows x 16 bytes per core matrix, 64-wide K chunks).
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace lmw {
namespace tc {

constexpr unsigned long long WAIT_NS = 2000000000ull;  // bound of every wait on an mbarrier (2 s)

__device__ __forceinline__ uint32_t su32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ uint64_t gtimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// true when the phase completed, false when the wait ran out after `ns` nanoseconds
__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t phase) {
  uint32_t done;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done)
               : "r"(bar), "r"(phase)
               : "memory");
  return done != 0;
}
// The timer is read only once a few tries (each of which the hardware suspends for a while) have failed: a wait that is
// soon over costs no timer read and no sleep
__device__ __forceinline__ bool wait_for(uint32_t bar, uint32_t phase, unsigned long long ns) {
  for (int k = 0; k < 32; k++)
    if (try_wait(bar, phase)) return true;
  const uint64_t t0 = gtimer();
  while (true) {
    if (try_wait(bar, phase)) return true;
    if (gtimer() - t0 > ns) return false;
    __nanosleep(20);
  }
}
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t phase) { return wait_for(bar, phase, WAIT_NS); }

// the same by a whole warp, with one outcome for all its lanes
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t phase) { return __all_sync(0xffffffffu, wait(bar, phase)) != 0; }

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// one bulk asynchronous copy (the TMA engine) of a contiguous run; both addresses 16-byte aligned, bytes a
// multiple of 16
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(bar)
               : "memory");
}

// shared-memory matrix descriptor of the chunk layout: K-direction core matrices 128 B apart, 8-row groups `sbo`
// bytes apart (1024 for chunks of 64 K columns, 16 x the chunk width in general), no swizzle, descriptor version 1
__device__ __forceinline__ uint64_t chunk_desc(uint32_t saddr, uint32_t sbo = 1024u) {
  uint64_t d = static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>(128u >> 4) << 16;
  d |= static_cast<uint64_t>(sbo >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}

// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M = 128, N
__device__ __forceinline__ uint32_t idesc_m128(int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
}

// The MMA role is a whole warp whose control flow is uniform, with the instruction predicated on one elected lane:
// descriptors and addresses then stay in uniform registers, where the instruction takes them from. Issued by a lone
// thread of a divergent branch, each MMA took about 115 cycles whatever its size.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ int uniform(int x) { return __shfl_sync(0xffffffffu, x, 0); }

__device__ __forceinline__ void mma(bool leader, uint32_t dtmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n .reg .pred p, q;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 q, %5, 0;\n @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
               "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate), "r"(static_cast<uint32_t>(leader))
               : "memory");
}
__device__ __forceinline__ void commit(bool leader, uint32_t bar) {
  asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
               "r"(static_cast<uint32_t>(leader))
               : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// allocation by one whole warp
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
}

// 8 consecutive accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void ld8(uint32_t taddr, float *v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

// 32 consecutive accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void ld32(uint32_t taddr, float *v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,"
      "%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

}  // namespace tc
}  // namespace lmw
