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

// How the CTAs of a cluster end when a wait has run out.  A message needs its
// receiver's shared memory, which lasts until the last warp of that CTA has
// gone, so no CTA may go while another can still send to it.
struct Leave {
  int dead;      // a wait of the cluster ran out
  int left;      // warps of this CTA that have gone or are about to
  int gone[16];  // by CTA: it has one warp left, which sends nothing more
};

// Before the cluster barrier that follows `init`.
__device__ __forceinline__ void leave_init(Leave& e) {
  if (threadIdx.x < 16) e.gone[threadIdx.x] = 0;
  if (threadIdx.x == 0) e.dead = e.left = 0;
}

// A store to the same word in CTA r.
__device__ __forceinline__ void store_to(int* p, int r, int v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(remote(p, r)), "r"(v)
               : "memory");
}

// The end of a warp (all its lanes) whose wait has run out, or that finds
// `dead` set after the kernel's last cluster barrier.  The CTAs are told first,
// so none of them can reach its own end without knowing.  Every warp but a CTA's
// last exits: barriers count threads that have exited as arrived, so the warps
// that still run get on, to a wait that runs out in turn or to the end.  The
// last warp takes part in the cluster's barriers until every CTA is down to its
// last warp; no message is sent any more then, and the pause lets those under
// way arrive.  (Out of line: it is long, and inlined at every wait it made the
// kernels slower; eight right-hand sides of the 3D 12x6x6 KKT 2.493 ms, 2.473 so,
// a direction of 2D SIMP 61x27 7.11 and 7.02.)
static __device__ __noinline__ void leave(Leave* e, int* status, int bit) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int cr, ncta;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cr));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ncta));
  if (lane < ncta) store_to(&e->dead, lane, 1);
  if (lane == 0) atomicOr(status, bit);
  __threadfence();
  __syncwarp();
  int before = 0;
  if (lane == 0) before = atomicAdd(&e->left, 1);
  if (__shfl_sync(FULL, before, 0) == (int)blockDim.x / 32 - 1) {
    if (lane < ncta) store_to(&e->gone[cr], lane, 1);
    volatile int* g = e->gone + (lane < ncta ? lane : 0);
    for (int it = 0; it < (1 << 20); it++) {
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\n"
                   "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
      if (__all_sync(FULL, *g)) break;
    }
    for (int i = 0; i < 64; i++) __nanosleep(1000);
  }
  asm volatile("exit;");
}

// Wait of a whole warp for a phase.  Bounded: when it runs out after `polls`
// polls, or `dead` is set (every message is sent before its receivers can need
// it, so only a fault elsewhere could make it), `bit` is set in *status and the
// warp leaves the kernel.
__device__ __forceinline__ void wait(unsigned long long* bar, unsigned parity, int polls,
                                     Leave& e, int* status, int bit) {
  for (int it = 0; it < polls; it++) {
    if (__reduce_min_sync(0xffffffffu, try_wait(bar, parity))) return;
    if ((it & 63) == 63 && __any_sync(0xffffffffu, *(volatile int*)&e.dead)) break;
  }
  leave(&e, status, bit);
}

}  // namespace msg
}  // namespace ab
