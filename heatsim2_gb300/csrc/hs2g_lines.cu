// A bounded device wait and its self-test: a wait on an mbarrier gives up after a limit of %globaltimer time and
// reports HS2G_ERR_TIMEOUT through its status word, leaving the context usable.  (The line solves are in hs2g_pair.cuh and
// hs2g_x.cuh; they have no such wait.)
#include "hs2g_internal.cuh"

namespace hs2g {
namespace {

__device__ __forceinline__ uint32_t saddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(saddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t deadline = now_ns() + limit_ns;
  while (!mbar_try_wait(bar, parity))
    if (now_ns() > deadline) return false;
  return true;
}
// Self-test of the bounded wait: one thread waits, for at most limit_ns, on an mbarrier that expects one
// arrival, which it makes itself (arrive != 0) or which never comes.  A wait that gives up reports
// HS2G_ERR_TIMEOUT through the status word; nothing is in flight, so the kernel ends cleanly either way.
__global__ void wait_selftest_kernel(uint64_t limit_ns, int arrive, int* status) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (arrive) mbar_arrive(&bar);
  *status = mbar_wait_bounded(&bar, 0, limit_ns) ? HS2G_OK : HS2G_ERR_TIMEOUT;
}

}  // namespace

cudaError_t wait_selftest(uint64_t limit_ns, int arrive, int* status_dev, cudaStream_t s) {
  wait_selftest_kernel<<<1, 32, 0, s>>>(limit_ns, arrive, status_dev);
  return cudaGetLastError();
}

}  // namespace hs2g
