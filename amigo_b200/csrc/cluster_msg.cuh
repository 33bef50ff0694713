// Messages between the CTAs of a thread-block cluster: stores into another
// CTA's shared memory that report their bytes to an mbarrier there (st.async),
// and the wait for them.  No fence and no cluster barrier stands between the
// value and its reader.  Measured on clusters of 8: 405 cycles for a release /
// acquire cluster barrier, 935 with one remote store per warp and CTA before
// it, ~200 for a message.
#pragma once
#include <cuda_runtime.h>

namespace ab {
namespace msg {

// The shared-memory address of `p` in CTA r of the cluster.
__device__ __forceinline__ unsigned remote(const void* p, int r) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  unsigned d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(r));
  return d;
}

__device__ __forceinline__ void send(unsigned dst, unsigned bar, float v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 "
               "[%0], %1, [%2];" ::"r"(dst), "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send(unsigned dst, unsigned bar, double v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 "
               "[%0], %1, [%2];" ::"r"(dst), "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send(unsigned dst, unsigned bar, uint4 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 "
               "[%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w), "r"(bar)
               : "memory");
}

// An mbarrier that one thread arms for each message (expect); the other CTAs
// may send to it after a cluster barrier that follows `init`.
__device__ __forceinline__ void init(unsigned long long* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(bar))
               : "memory");
}
__device__ __forceinline__ void init_done() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void expect(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(bar)),
               "r"(bytes)
               : "memory");
}

// Whether phase `parity` of the mbarrier is complete (waits a short while).
__device__ __forceinline__ unsigned try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"((unsigned)__cvta_generic_to_shared(bar)), "r"(parity)
      : "memory");
  return ok;
}

// Wait of a whole warp for a phase.  Bounded: when it runs out (every message
// is sent before its receivers can need it, so only a fault elsewhere could
// make it) `bit` is set in *status and the warp leaves the kernel; the CTA's
// and the cluster's barriers count threads that have left as arrived, so the
// other warps end too.
__device__ __forceinline__ void wait(unsigned long long* bar, unsigned parity, int* status,
                                     int bit) {
  for (int it = 0; it < (1 << 20); it++)
    if (__reduce_min_sync(0xffffffffu, try_wait(bar, parity))) return;
  atomicOr(status, bit);
  __threadfence();
  asm volatile("exit;");
}

}  // namespace msg
}  // namespace ab
