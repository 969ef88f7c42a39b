// Shared by the tcgen05 kernels of the prompt path: bounded mbarrier waits, descriptors, tensor-memory loads and stores.
#pragma once
#include "common.cuh"

namespace b200 {
namespace umma {

// Polls before a wait gives up: about a second (a poll that is not met suspends the warp for 7,760 clocks). Counted and not timed: the
// clock runs on while the GPU is given to another process, and a wait that is about to be met must not end for that.
constexpr int kSpin = 1 << 18;

DEVI uint32_t sa(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
DEVI void bar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sa(b)), "r"(count));
}
DEVI void bar_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa(b)) : "memory"); }
DEVI uint32_t in_cta(uint32_t local, uint32_t rank) {   // the same shared-memory offset in CTA `rank` of the cluster
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
// Arrivals and waits carry no cluster-scope fence: what they order is tensor memory (the tcgen05 fences beside them) and bulk
// copies (their own transaction counts); an acquire at cluster scope would empty the L1 on every poll.
DEVI void bar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
DEVI bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(sa(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// false if the phase did not complete within the bound or another role of the CTA has given up; *status <- code of the first wait
// that ran out
template <int SLEEP_NS>
DEVI bool bar_wait(uint64_t* b, uint32_t parity, volatile int* fail, int* status, int code) {
  if (bar_try(b, parity)) return true;
#pragma unroll 1
  for (int i = 0; i < kSpin; ++i) {
    if (SLEEP_NS > 0) __nanosleep(SLEEP_NS);
    if (bar_try(b, parity)) return true;
    if ((i & 63) == 63 && *fail) return false;
  }
  *fail = 1;
  atomicCAS(status, 0, code);
  return false;
}
DEVI void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
DEVI float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// The power of two p with m < p <= 2 m, within 2^-59 .. 2^41 (0: the smallest, infinity: the largest).
DEVI float pow2_above(float m) {
  const int e = (int)((__float_as_uint(m) >> 23) & 255u) + 1;
  return __int_as_float(min(max(e, 68), 168) << 23);
}
// Shared-memory matrix descriptor, 128-byte swizzle, rows of 128 bytes, eight rows per 1024-byte block. K-major operand: rows are M or
// N, 64 fp16 of K each; `lead` unused (1). MN-major operand: rows are K, 64 fp16 of M or N each; `lead` = bytes from one 64-wide block
// of M or N to the next.
DEVI uint64_t desc_sw128(uint32_t addr, uint32_t lead = 16) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lead >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

DEVI void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr)
      : "memory");
}
DEVI void tmem_ld8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "r"(addr)
      : "memory");
}
DEVI void tmem_st8(uint32_t addr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// without the wait; v is valid after tmem_wait_ld()
DEVI void tmem_ld16_async(uint32_t addr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
                 "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
               : "r"(addr)
               : "memory");
}
// the values of earlier tmem_ld16_async calls pass through, so that nothing is computed from them before the wait
template <int N>
DEVI void tmem_wait_ld(float (&v)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+f"(v[i]));
}
DEVI void tmem_st16(uint32_t addr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

}  // namespace umma
}  // namespace b200
