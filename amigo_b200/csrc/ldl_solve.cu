// Triangular solves with the multifrontal LDL^T factor (FP64).
//
// Forward sweep (levels ascending; a CTA, a cluster or the grid per front, by
// size): the front vector is
// assembled from the right-hand side of the node's own variables plus the
// update vectors of its children, placed by the same row map as the
// factorization's extend-add; L11 is applied in column blocks (one warp
// solves a block, the CTA updates the rows below it), the tail is kept as
// this front's update vector for the parent, and D^{-1} (1x1 / 2x2 blocks)
// gives the pivots' values.  Backward sweep (levels descending): the front
// gathers the final values of its delayed and contribution rows, applies
// L21^T and L11^T and writes its pivots.  The arithmetic is that of the
// reference's solve_ldl (include/sparse_ldl.h:1807-1908,
// solve_pivot_lower/diagonal/transpose 1550-1669) reorganised so that fronts
// of one level run concurrently without atomics.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <utility>
#include <vector>

#include "cluster_msg.cuh"
#include "ldl_internal.h"
#include "launch_count.h"

namespace ab {
namespace {

constexpr int NT = kThreads;
constexpr int SB = 32;  // column block of the triangular solves

__device__ __forceinline__ int decode_var(int v) { return v >= 0 ? v : -v - 1; }

// Block end for pivot columns starting at jb: at most SB columns and never
// splitting a 2x2 pair (kind 1 = first column of a pair).
__device__ __forceinline__ int block_end(const int* kind, int jb, int npiv) {
  int je = jb + SB < npiv ? jb + SB : npiv;
  if (je < npiv && kind[je - 1] == 1) je++;
  return je;
}

// sum_{j < n} col[j * ld] * v(j), accumulated in the order of j, with the
// loads issued 16 at a time so that they overlap (the factor streams from
// HBM / L2 with hundreds of cycles of latency per load).
template <class T, class VF>
__device__ __forceinline__ double dot_strided(const T* __restrict__ col, size_t ld,
                                              int n, VF v) {
  double acc = 0.0;
  int j = 0;
  for (; j + 16 <= n; j += 16) {
    T a[16];
#pragma unroll
    for (int u = 0; u < 16; u++) a[u] = col[(size_t)(j + u) * ld];
#pragma unroll
    for (int u = 0; u < 16; u++) acc = __fma_rn((double)a[u], v(j + u), acc);
  }
  for (; j < n; j++) acc = __fma_rn((double)col[(size_t)j * ld], v(j), acc);
  return acc;
}

// One lane's share of sum_{i0 <= i < i1} col[i] v(i): rows i0 + lane + 32 t
// in the order of t, with the loads issued 8 at a time.
template <class T, class VF>
__device__ __forceinline__ double lane_dot(const T* __restrict__ col, int i0, int i1,
                                           int lane, VF v) {
  double acc = 0.0;
  int i = i0 + lane;
  for (; i + 7 * 32 < i1; i += 8 * 32) {
    T a[8];
    double b[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      a[u] = col[i + 32 * u];
      b[u] = v(i + 32 * u);
    }
#pragma unroll
    for (int u = 0; u < 8; u++) acc = __fma_rn((double)a[u], b[u], acc);
  }
  for (; i < i1; i += 32) acc = __fma_rn((double)col[i], v(i), acc);
  return acc;
}

// The 2x2 block of D applied to (x1, x2): every product and difference
// rounded on its own (no contraction), so that every kernel that solves
// with a 2x2 pivot gives the same bits.
__device__ __forceinline__ double inv2x2(double d11, double d21, double d22) {
  return __ddiv_rn(1.0, __dsub_rn(__dmul_rn(d11, d22), __dmul_rn(d21, d21)));
}
__device__ __forceinline__ double piv2_first(double inv, double d21, double d22,
                                             double x1, double x2) {
  return __dmul_rn(inv, __dsub_rn(__dmul_rn(d22, x1), __dmul_rn(d21, x2)));
}
__device__ __forceinline__ double piv2_second(double inv, double d11, double d21,
                                              double x1, double x2) {
  return __dmul_rn(inv, __dsub_rn(__dmul_rn(d11, x2), __dmul_rn(d21, x1)));
}

__device__ __forceinline__ double warp_sum_down(double a) {
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  return a;
}

// The value of row j of a block held R rows per lane (row lane + 32 r in
// v[r]), broadcast to the warp.
template <int R>
__device__ __forceinline__ double warp_row(const double (&v)[R], int j) {
  double s = v[0];
#pragma unroll
  for (int r = 1; r < R; r++)
    if ((j >> 5) == r) s = v[r];
  return __shfl_sync(0xffffffffu, s, j & 31);
}

// One warp solves the unit lower triangle of a diagonal block (bw <= 32 R
// rows, column-major in sL with leading dimension lds, pivot kinds in sK)
// in place on V[0:bw], with the block's values in registers: each step is
// one broadcast and one multiply-add per row.  A 2x2 pair (kind 1, 2)
// eliminates both columns at once; its off-diagonal entry belongs to D.
template <int R>
__device__ __forceinline__ void warp_lower_solve(const double* sL, int lds,
                                                 const int* sK, int bw, double* V,
                                                 int lane) {
  double v[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int i = lane + 32 * r;
    v[r] = i < bw ? V[i] : 0.0;
  }
  for (int j = 0; j < bw;) {
    const bool two = sK[j] == 1;
    const double v0 = warp_row<R>(v, j);
    const double v1 = two ? warp_row<R>(v, j + 1) : 0.0;
    const int i0 = j + (two ? 2 : 1);
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int i = lane + 32 * r;
      if (i >= i0 && i < bw) {
        double t = __dmul_rn(sL[i + j * lds], v0);
        if (two) t = __fma_rn(sL[i + (j + 1) * lds], v1, t);
        v[r] = __dsub_rn(v[r], t);
      }
    }
    j = i0;
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int i = lane + 32 * r;
    if (i < bw) V[i] = v[r];
  }
}

// One warp solves the unit upper triangle L^T of a diagonal block in place
// on V[0:bw], from the last pivot backwards: once a pivot's value is final
// it is broadcast and every earlier row subtracts its term.
template <int R>
__device__ __forceinline__ void warp_upper_solve(const double* sL, int lds,
                                                 const int* sK, int bw, double* V,
                                                 int lane) {
  double v[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int i = lane + 32 * r;
    v[r] = i < bw ? V[i] : 0.0;
  }
  for (int j = bw - 1; j >= 0;) {
    const bool two = sK[j] == 2;
    const int jl = two ? j - 1 : j;
    const double xj = warp_row<R>(v, j);
    const double xl = two ? warp_row<R>(v, jl) : 0.0;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int i = lane + 32 * r;
      if (i < jl) {
        double t = __dmul_rn(sL[j + i * lds], xj);
        if (two) t = __fma_rn(sL[jl + i * lds], xl, t);
        v[r] = __dsub_rn(v[r], t);
      }
    }
    j = jl - 1;
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int i = lane + 32 * r;
    if (i < bw) V[i] = v[r];
  }
}

// Programmatic dependent launch (see the factorization's pdl_enter): wait
// for the previous kernel of the stream, then let the next be scheduled.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Front vector of `node` for one right-hand side: the node's own entries
// of the right-hand side plus the update vectors of its children, placed
// by the same row map as the factorization's extend-add.  Called by a
// whole CTA; V may be shared or global memory.
template <int NTH = NT>
__device__ void assemble_front_vector(const DevicePlan& d, int node, double* V,
                                      const double* xr, const double* ubuf,
                                      const long long* uoff, int rhs,
                                      int* s_choff) {
  const int tid = threadIdx.x;
  const int f = d.f[node];
  const int ns = d.ns[node], ndin = d.ndin[node];
  const int fs = ns + ndin;
  const int* fsinv = d.ipool + d.ioff[node] + 2 * f;
  for (int r = tid; r < f; r += NTH) V[r] = 0.0;
  __syncthreads();
  const int vb = d.var_ptr[node];
  for (int r = tid; r < ns; r += NTH) V[fsinv[r]] = xr[d.vars[vb + r]];
  __syncthreads();
  if (tid == 0) *s_choff = ns;
  __syncthreads();
  for (int q = d.kid_ptr[node]; q < d.kid_ptr[node + 1]; q++) {
    const int c = d.kids[q];
    const int fc = d.f[c], npc = d.npiv[c], ndc = d.ndel[c];
    const int cc = fc - npc;
    const double* uc = ubuf + uoff[c] + (long long)rhs * fc + npc;
    const int cb = d.cptr[c];
    const int choff = *s_choff;
    for (int a = tid; a < cc; a += NTH) {
      int pos;
      if (a < ndc) {
        pos = choff + a;
      } else {
        int r0 = d.cmap[cb + a - ndc];
        pos = r0 < ns ? r0 : r0 + ndin;
      }
      if (pos < fs) pos = fsinv[pos];
      V[pos] += __ldcg(uc + a);  // written by another CTA (queue sweeps)
    }
    __syncthreads();
    if (tid == 0) *s_choff = choff + ndc;
    __syncthreads();
  }
}

// Shared scratch of the one-CTA front solves.
struct NarrowSmem {
  int choff;
  double L[(SB + 1) * (SB + 1)];
  int K[SB + 1];  // the block's pivot kinds
};

// Forward solve of one front by the whole CTA (sV: dynamic shared memory
// of smem_doubles).
template <class T, int NTH = NT>
__device__ void forward_front(const DevicePlan& d, int node, double* x, int nrhs,
                              int ldx, double* ubuf, const long long* uoff,
                              int smem_doubles, double* sV, NarrowSmem& sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = d.f[node], npiv = d.npiv[node];
  const int* fvars = d.ipool + d.ioff[node];
  const int* kind = fvars + 3 * f;
  const T* L = reinterpret_cast<const T*>(d.fpool) + d.foff[node];
  int& s_choff = sm.choff;
  double* sL = sm.L;
  int* sK = sm.K;

  for (int rhs = blockIdx.y; rhs < nrhs; rhs += gridDim.y) {
    // The front vector is worked on in shared memory when it fits (every
    // step of the in-block triangular solve depends on the previous one);
    // its tail is stored in ubuf for the parent.
    double* G = ubuf + uoff[node] + (long long)rhs * f;
    double* V = f <= smem_doubles ? sV : G;
    double* xr = x + (long long)rhs * ldx;
    assemble_front_vector<NTH>(d, node, V, xr, ubuf, uoff, rhs, &s_choff);

    // Forward elimination with the unit lower factor.  The diagonal block
    // of each column block is staged in shared memory first, so that the
    // dependent steps of the warp's triangular solve read no global memory.
    for (int jb = 0; jb < npiv;) {
      const int je = block_end(kind, jb, npiv);
      const int bw = je - jb;
      for (int t = tid; t < bw * bw; t += NTH) {
        const int i = t % bw, j = t / bw;
        sL[i + j * (SB + 1)] = L[jb + i + (size_t)(jb + j) * f];
      }
      for (int t = tid; t < bw; t += NTH) sK[t] = kind[jb + t];
      __syncthreads();
      if (warp == 0) warp_lower_solve<2>(sL, SB + 1, sK, bw, V + jb, lane);
      __syncthreads();
      for (int i = je + tid; i < f; i += NTH)
        V[i] -= dot_strided(L + i + (size_t)jb * f, (size_t)f, bw,
                            [&](int j) { return V[jb + j]; });
      __syncthreads();
      jb = je;
    }
    // D^{-1} and the pivots' forward values.
    for (int j = tid; j < npiv; j += NTH) {
      const int kd = kind[j];
      if (kd == 0) {
        V[j] = V[j] / L[j + (size_t)j * f];
      } else if (kd == 1) {
        const double d11 = L[j + (size_t)j * f];
        const double d21 = L[j + 1 + (size_t)j * f];
        const double d22 = L[j + 1 + (size_t)(j + 1) * f];
        const double inv = inv2x2(d11, d21, d22);
        const double x1 = V[j], x2 = V[j + 1];
        V[j] = piv2_first(inv, d21, d22, x1, x2);
        V[j + 1] = piv2_second(inv, d11, d21, x1, x2);
      }
    }
    __syncthreads();
    for (int j = tid; j < npiv; j += NTH) xr[decode_var(fvars[j])] = V[j];
    if (V != G)
      for (int r = npiv + tid; r < f; r += NTH) G[r] = V[r];
    __syncthreads();
  }
}

#include "solve_front.cuh"

// Whether a narrow front's pivot columns go to the launch's shared memory.
template <class T>
__device__ __forceinline__ bool solve_staged(const DevicePlan& d, int node, int smem_doubles) {
  return staged_bytes<T>(d.f[node], d.npiv[node]) <= 8 * (size_t)smem_doubles &&
         !(d.general_forms & 2);
}

template <class T, int NTH = NT>
__global__ void __launch_bounds__(NTH)
k_solve_forward(DevicePlan d, const int* __restrict__ nodes, double* x,
                int nrhs, int ldx, double* ubuf, const long long* uoff,
                int smem_doubles) {
  pdl_enter();
  extern __shared__ double sV[];
  __shared__ NarrowSmem sm;
  const int node = nodes[blockIdx.x];
  if (solve_staged<T>(d, node, smem_doubles))
    forward_staged<T, NTH>(d, node, x, nrhs, ldx, ubuf, uoff, reinterpret_cast<char*>(sV),
                           []() {});
  else
    forward_front<T, NTH>(d, node, x, nrhs, ldx, ubuf, uoff, smem_doubles, sV, sm);
}

// Backward solve of one front by the whole CTA.
template <class T, int NTH = NT>
__device__ void backward_front(const DevicePlan& d, int node, double* x, int nrhs,
                               int ldx, double* ubuf, const long long* uoff,
                               int smem_doubles, double* sV, NarrowSmem& sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWARP = NTH / 32;
  const int f = d.f[node], npiv = d.npiv[node];
  const int* fvars = d.ipool + d.ioff[node];
  const int* kind = fvars + 3 * f;
  const T* L = reinterpret_cast<const T*>(d.fpool) + d.foff[node];
  double* sL = sm.L;
  int* sK = sm.K;
  for (int rhs = blockIdx.y; rhs < nrhs; rhs += gridDim.y) {
    double* V = f <= smem_doubles ? sV : ubuf + uoff[node] + (long long)rhs * f;
    double* xr = x + (long long)rhs * ldx;
    // pivots: their forward values (written to x by the forward sweep);
    // delayed and contribution rows: final values of the ancestors (from
    // L2: another CTA of the same sweep may have written them)
    for (int r = tid; r < npiv; r += NTH) V[r] = xr[decode_var(fvars[r])];
    for (int r = npiv + tid; r < f; r += NTH) V[r] = __ldcg(xr + fvars[r]);
    __syncthreads();
    // Column blocks from the last one backwards.
    int je = npiv;
    while (je > 0) {
      int jb = je - SB > 0 ? je - SB : 0;
      if (jb > 0 && kind[jb] == 2) jb--;  // keep 2x2 pairs together
      // t[j] -= sum_{i >= je} L[i, j] t[i] for j in [jb, je): one warp per
      // column, lanes over rows.
      for (int j = jb + warp; j < je; j += NWARP) {
        const double acc = warp_sum_down(
            lane_dot(L + (size_t)j * f, je, f, lane, [&](int i) { return V[i]; }));
        if (lane == 0) V[j] -= acc;
      }
      const int bw = je - jb;
      for (int t = tid; t < bw * bw; t += NTH) {
        const int i = t % bw, j = t / bw;
        sL[i + j * (SB + 1)] = L[jb + i + (size_t)(jb + j) * f];
      }
      for (int t = tid; t < bw; t += NTH) sK[t] = kind[jb + t];
      __syncthreads();
      // within the block, backwards: column j (or pair j-1, j)
      if (warp == 0) warp_upper_solve<2>(sL, SB + 1, sK, bw, V + jb, lane);
      __syncthreads();
      je = jb;
    }
    for (int j = tid; j < npiv; j += NTH) xr[decode_var(fvars[j])] = V[j];
    __syncthreads();
  }
}

template <class T, int NTH = NT>
__global__ void __launch_bounds__(NTH)
k_solve_backward(DevicePlan d, const int* __restrict__ nodes, double* x,
                 int nrhs, int ldx, double* ubuf, const long long* uoff,
                 int smem_doubles) {
  pdl_enter();
  extern __shared__ double sV[];
  __shared__ NarrowSmem sm;
  const int node = nodes[blockIdx.x];
  if (solve_staged<T>(d, node, smem_doubles))
    backward_staged<T, NTH>(d, node, x, nrhs, ldx, reinterpret_cast<char*>(sV), []() {});
  else
    backward_front<T, NTH>(d, node, x, nrhs, ldx, ubuf, uoff, smem_doubles, sV, sm);
}

// Narrow fronts of at most kSmallRows rows run on CTAs of kSmallThreads
// threads (more fronts in flight per SM; the same steps in the same order,
// so the same bits).
constexpr int kSmallRows = 128;
constexpr int kSmallThreads = 128;

// ---------------------------------------------------------------------------
// Work-queue sweeps over the levels whose fronts are all narrow: one launch
// per sweep instead of one per level.  `nodes` lists the fronts in the
// order of a sweep (forward: level by level from the leaves; backward: the
// reverse); each CTA takes the next front from an atomic counter, waits
// until the fronts it depends on are done (forward: its children;
// backward: its parent, when the parent is in the queue), solves it and
// marks it done with this sweep's epoch.  Fronts are handed out in
// dependency order and a CTA takes a front only while it runs, so the
// earliest unfinished front always has its dependencies done: the waits
// end.  Each wait is still bounded; when one runs out the kernel records
// it in *err (the host reports it) and goes on.
constexpr long long kQueuePolls = 1ll << 22;

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void wait_done(const unsigned* flag, unsigned epoch, int* err) {
  for (long long it = 0; it < kQueuePolls; it++) {
    if (ld_acquire(flag) == epoch) return;
    if (it >= 16) __nanosleep(64);
  }
  atomicOr(err, 1);
}

// Take the next queue entry (-1 when the queue is exhausted).
__device__ __forceinline__ int queue_next(unsigned* ctr, int count, int* s_idx) {
  __syncthreads();
  if (threadIdx.x == 0) *s_idx = (int)atomicAdd(ctr, 1u);
  __syncthreads();
  const int idx = *s_idx;
  return idx < count ? idx : -1;
}

// This front's results are visible GPU-wide before its done flag.
__device__ __forceinline__ void mark_done(unsigned* flag, unsigned epoch) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) st_release(flag, epoch);
}

// Start of a solve's two queued sweeps: zero the queue counters (forward and
// backward of every right-hand-side slice) and move to the next epoch.  The epoch lives in device memory, so a
// captured CUDA graph of a solve takes a new epoch on every replay.
constexpr int kEpochWord = 2 * kRhsSlices;
__global__ void k_sweep_begin(unsigned* ctr) {
  if (threadIdx.x < 2 * kRhsSlices) ctr[threadIdx.x] = 0u;
  if (threadIdx.x == 0) ctr[kEpochWord] = ctr[kEpochWord] + 1u;
}

template <class T, int NTH = NT>
__global__ void __launch_bounds__(NTH)
k_solve_forward_q(DevicePlan d, const int* __restrict__ nodes, int count, double* x,
                  int nrhs, int ldx, double* ubuf, const long long* uoff,
                  int smem_doubles, unsigned* ctr, unsigned* done, const unsigned* ep,
                  int* err) {
  pdl_enter();
  extern __shared__ double sV[];
  __shared__ NarrowSmem sm;
  __shared__ int s_idx;
  ctr += blockIdx.y;
  done += (size_t)blockIdx.y * d.nn;
  const unsigned epoch = *ep;
  for (;;) {
    const int idx = queue_next(ctr, count, &s_idx);
    if (idx < 0) break;
    const int node = nodes[idx];
    auto wait = [&]() {
      for (int q = d.kid_ptr[node] + threadIdx.x; q < d.kid_ptr[node + 1]; q += NTH)
        wait_done(done + d.kids[q], epoch, err);
    };
    if (solve_staged<T>(d, node, smem_doubles)) {
      forward_staged<T, NTH>(d, node, x, nrhs, ldx, ubuf, uoff, reinterpret_cast<char*>(sV),
                             wait);
    } else {
      wait();
      __syncthreads();
      forward_front<T, NTH>(d, node, x, nrhs, ldx, ubuf, uoff, smem_doubles, sV, sm);
    }
    mark_done(done + node, epoch);
  }
}

template <class T, int NTH = NT>
__global__ void __launch_bounds__(NTH)
k_solve_backward_q(DevicePlan d, const int* __restrict__ nodes,
                   const int* __restrict__ dep, int count, double* x, int nrhs,
                   int ldx, double* ubuf, const long long* uoff, int smem_doubles,
                   unsigned* ctr, unsigned* done, const unsigned* ep, int* err) {
  pdl_enter();
  extern __shared__ double sV[];
  __shared__ NarrowSmem sm;
  __shared__ int s_idx;
  ctr += blockIdx.y;
  done += (size_t)blockIdx.y * d.nn;
  const unsigned epoch = *ep;
  for (;;) {
    const int idx = queue_next(ctr, count, &s_idx);
    if (idx < 0) break;
    const int node = nodes[idx];
    auto wait = [&]() {
      if (threadIdx.x == 0 && dep[idx] >= 0) wait_done(done + dep[idx], epoch, err);
    };
    if (solve_staged<T>(d, node, smem_doubles)) {
      backward_staged<T, NTH>(d, node, x, nrhs, ldx, reinterpret_cast<char*>(sV), wait);
    } else {
      wait();
      __syncthreads();
      backward_front<T, NTH>(d, node, x, nrhs, ldx, ubuf, uoff, smem_doubles, sV, sm);
    }
    mark_done(done + node, epoch);
  }
}


// ---------------------------------------------------------------------------
// Mid-size fronts: one thread-block cluster of CS CTAs per front.  CTA 0
// solves the pivot block, a chain of 32-column blocks; the contribution rows'
// product with it (the update vector passed to the parent, forward; the
// pivots' right-hand side correction, backward) is spread over the other CTAs,
// which read the front's L21 once.  The two overlap: forward, a block's values
// are sent to the other CTAs as soon as they are known; backward, the other
// CTAs send the columns' corrections, last block first, and CTA 0 takes a block
// when its columns are there.  Everything that does not depend on another
// front's values is fetched before the previous launch of the solve is done
// (the factor was finished before the solve's first launch, see launch_solve).
constexpr int CS = 8;

constexpr int CW = CS - 1;                // CTAs that take the contribution rows
constexpr int DB = (SB + 1) * (SB + 1);   // a diagonal block
constexpr int kCluKids = 8;               // children whose sizes are held
constexpr int kCluWait = 2;               // error word bit: a message's wait ran out

// Shared memory of a cluster front: its vector (CTA 0; backward the pivots'
// values and their corrections) or the pivots' values and sums of rows past 256
// (the other CTAs; backward the contribution rows' values), two diagonal blocks, an mbarrier per block, the children's row
// positions, the blocks' first columns and the pivot kinds.
struct CluSmem {
  double* V;
  double* diag;              // 2 x DB
  unsigned long long* bar;   // a block each
  int* P;                    // clu_positions(f)
  unsigned short* jb;        // blocks + 1
  unsigned char* K;
};
// Row positions held (past 8,192 rows the vector takes their room).
__host__ __device__ __forceinline__ int clu_positions(int f) { return f <= 8192 ? 2 * f : 0; }
__host__ __device__ __forceinline__ int clu_blocks(int npiv) { return npiv / (SB - 1) + 2; }
__host__ __device__ __forceinline__ int clu_vector(int f, int npiv) {
  return f > 2 * npiv ? f : 2 * npiv;
}
__host__ __device__ __forceinline__ size_t clu_bytes(int f, int npiv) {
  return ((size_t)clu_vector(f, npiv) + 2 * DB + clu_blocks(npiv)) * 8 +
         (size_t)clu_positions(f) * 4 + 2 * (size_t)clu_blocks(npiv) + npiv + 16;
}
__device__ __forceinline__ CluSmem clu_smem(double* raw, int f, int npiv) {
  CluSmem m;
  m.V = raw;
  m.diag = raw + clu_vector(f, npiv);
  m.bar = reinterpret_cast<unsigned long long*>(m.diag + 2 * DB);
  m.P = reinterpret_cast<int*>(m.bar + clu_blocks(npiv));
  m.jb = reinterpret_cast<unsigned short*>(m.P + clu_positions(f));
  m.K = reinterpret_cast<unsigned char*>(m.jb + clu_blocks(npiv));
  return m;
}

// The diagonal block of columns [jb, jb + bw) into `dst` (in flight until
// cp_wait); T entries, leading dimension SB + 1.
template <class T>
__device__ __forceinline__ void fetch_diag(const T* L, int f, int jb, int bw, double* dst) {
  T* o = reinterpret_cast<T*>(dst);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = warp; j < bw; j += NT / 32)
    for (int i = lane; i < bw; i += 32)
      if (i >= j) cp_async_el(o + i + j * (SB + 1), L + jb + i + (size_t)(jb + j) * f);
}

// Pivot kinds and blocks of a front (every CTA), and its mbarriers; returns
// the number of blocks.  forward: blocks from the first column on (block_end),
// else from the last one backwards.
__device__ __forceinline__ int clu_setup(const CluSmem& m, const int* kind, int npiv,
                                         bool forward, int* s_nb, msg::Leave& leave) {
  const int tid = threadIdx.x;
  for (int j = tid; j < npiv; j += NT) m.K[j] = (unsigned char)kind[j];
  for (int b = tid; b < clu_blocks(npiv); b += NT) msg::init(m.bar + b);
  msg::leave_init(leave);
  msg::init_done();
  __syncthreads();
  if (tid == 0) {
    // first columns in the order of the sweep, then its end
    int nb = 0, j = forward ? 0 : npiv;
    while (forward ? j < npiv : j > 0) {
      m.jb[nb++] = (unsigned short)j;
      if (forward) {
        int je = min(j + SB, npiv);
        if (je < npiv && m.K[je - 1] == 1) je++;
        j = je;
      } else {
        int jb = max(j - SB, 0);
        if (jb > 0 && m.K[jb] == 2) jb--;  // keep 2x2 pairs together
        j = jb;
      }
    }
    m.jb[nb] = (unsigned short)j;
    *s_nb = nb;
  }
  __syncthreads();
  return *s_nb;
}

// CTA 0 carries the pivot chain: a block's diagonal is in shared memory and its
// entries of the next 256 rows in registers before its turn comes, so a block
// costs one warp's triangular solve and 32 multiply-adds a row, without a global
// load in between.  The other seven CTAs hold the rows below the pivots; CTA 0
// sends them each block's solution as messages (cluster_msg.cuh), so they work
// on a block while CTA 0 is at the next and no cluster barrier stands between
// blocks (405 cycles each, 935 after remote stores).  One solve of the 2D SIMP
// 128x64 KKT (fronts of ~1,100 rows and ~280 pivots, one after another): 3.77 ms
// with every CTA's entries fetched from global memory at its turn, 2.44 with the
// fetches ahead and a cluster barrier a block, 2.02 with the messages.
template <class T>
__global__ void __launch_bounds__(NT, 1)
k_clu_forward(DevicePlan d, const int* __restrict__ nodes, double* x, int nrhs, int ldx,
              double* ubuf, const long long* uoff, int* err) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ double sm[];
  __shared__ int s_nb;
  __shared__ msg::Leave s_leave;
  __shared__ int s_kid[kCluKids], s_cc[kCluKids];
  __shared__ long long s_uc[kCluKids];
  const int cr = (int)cluster.block_rank();
  const int node = nodes[blockIdx.x / CS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = d.f[node], npiv = d.npiv[node];
  const int* fvars = d.ipool + d.ioff[node];
  const T* L = reinterpret_cast<const T*>(d.fpool) + d.foff[node];
  const CluSmem m = clu_smem(sm, f, npiv);
  double* V = m.V;
  const int ns = d.ns[node], ndin = d.ndin[node], fs = ns + ndin;
  const int* fsinv = fvars + 2 * f;
  const int q0 = d.kid_ptr[node], nk = d.kid_ptr[node + 1] - q0;
  const int nb = clu_setup(m, fvars + 3 * f, npiv, true, &s_nb, s_leave);
  auto position = [&](int c, int ndc, int choff, int a) {
    int pos;
    if (a < ndc) {
      pos = choff + a;
    } else {
      const int r0 = d.cmap[d.cptr[c] + a - ndc];
      pos = r0 < ns ? r0 : r0 + ndin;
    }
    return pos < fs ? fsinv[pos] : pos;
  };
  int held = 0;  // children whose rows' positions are held
  const int vb = d.var_ptr[node];
  if (cr == 0) {
    if (tid < min(nk, kCluKids)) {
      const int c = d.kids[q0 + tid];
      s_kid[tid] = c;
      s_cc[tid] = d.f[c] - d.npiv[c];
      s_uc[tid] = uoff[c];
    }
    for (int q = 0, choff = ns, at = 0; q < min(nk, kCluKids); q++) {
      const int c = d.kids[q0 + q], ndc = d.ndel[c], cc = d.f[c] - d.npiv[c];
      if (at + cc > clu_positions(f)) break;
      for (int a = tid; a < cc; a += NT) m.P[at + a] = position(c, ndc, choff, a);
      at += cc;
      choff += ndc;
      held = q + 1;
    }
  }
  // the other CTAs' rows: 32-row strips dealt over them, a row a thread (and
  // every 256th after it)
  const int nstrip = (f - npiv + 31) / 32;
  auto row_of = [&](int t) { return npiv + ((cr - 1) + CW * (t >> 5)) * 32 + (t & 31); };
  const int nrow = cr > 0 ? 32 * ((nstrip - (cr - 1) + CW - 1) / CW) : 0;
  if (cr > 0)
    for (int b = tid; b < nb; b += NT)
      msg::expect(m.bar + b, 8u * (unsigned)(m.jb[b + 1] - m.jb[b]));
  // the columns' products are summed in eight segments, added in order
  const int seg = (npiv + 7) / 8;
  cluster.sync();
  pdl_enter();
  unsigned phase = 0;
  for (int rhs = blockIdx.y; rhs < nrhs; rhs += gridDim.y) {
    double* G = ubuf + uoff[node] + (long long)rhs * f;
    double* xr = x + (long long)rhs * ldx;
    if (cr == 0) {
      for (int r = tid; r < f; r += NT) V[r] = 0.0;
      if (nb > 0) fetch_diag<T>(L, f, 0, m.jb[1], m.diag);
      __syncthreads();
      for (int r = tid; r < ns; r += NT) V[fsinv[r]] = xr[d.vars[vb + r]];
      __syncthreads();
      for (int q = 0, choff = ns, at = 0; q < nk; q++) {
        const int c = q < kCluKids ? s_kid[q] : d.kids[q0 + q];
        const int cc = q < kCluKids ? s_cc[q] : d.f[c] - d.npiv[c];
        const double* uc = ubuf + (q < kCluKids ? s_uc[q] : uoff[c]) +
                           (long long)rhs * d.f[c] + d.npiv[c];
        const int ndc = d.ndel[c];
        for (int a = tid; a < cc; a += NT)
          V[q < held ? m.P[at + a] : position(c, ndc, choff, a)] += __ldcg(uc + a);
        __syncthreads();
        at += cc;
        choff += ndc;
      }
      for (int b = 0; b < nb; b++) {
        const int jb = m.jb[b], je = m.jb[b + 1], bw = je - jb;
        const T* D = reinterpret_cast<const T*>(m.diag + (b & 1) * DB);
        // warp 0 solves; the other warps load the block's entries of the next
        // 224 rows (a row a thread, the 33rd column apart) and the next
        // diagonal block meanwhile
        const int i0 = warp > 0 ? je + tid - 32 : npiv;
        T a[SB], a32 = T(0);
        cp_wait();
        __syncthreads();  // the diagonal block; the rows' updates of the last one
        if (warp == 0) {
          lower_block<T>(D, SB + 1, m.K + jb, bw, V + jb, lane);
        } else {
          const T* Li = L + (i0 < npiv ? i0 : 0) + (size_t)jb * f;
#pragma unroll
          for (int j = 0; j < SB; j++) a[j] = i0 < npiv && j < bw ? Li[(size_t)j * f] : T(0);
          if (bw > SB && i0 < npiv) a32 = Li[(size_t)SB * f];
        }
        if (b + 1 < nb)
          fetch_diag<T>(L, f, je, m.jb[b + 2] - je, m.diag + ((b + 1) & 1) * DB);
        __syncthreads();
        if (warp == NT / 32 - 1 && nstrip > 0) {
          // the block's values to the other CTAs
          for (int j = lane; j < bw; j += 32)
#pragma unroll
            for (int r = 1; r < CS; r++)
              msg::send(msg::remote(V + jb + j, r), msg::remote(m.bar + b, r), V[jb + j]);
        }
        if (warp == NT / 32 - 2) {
          // D^{-1} and the pivots' forward values
          for (int j = lane; j < bw; j += 32) {
            const int kd = m.K[jb + j];
            double v;
            if (kd == 0) {
              v = V[jb + j] / (double)D[j * (SB + 2)];
            } else {
              const T* Df = D + (j - kd + 1) * (SB + 2);  // the pair's first diagonal
              const double d11 = Df[0], d21 = Df[1], d22 = Df[SB + 2];
              const double inv = inv2x2(d11, d21, d22);
              v = kd == 1 ? piv2_first(inv, d21, d22, V[jb + j], V[jb + j + 1])
                          : piv2_second(inv, d11, d21, V[jb + j - 1], V[jb + j]);
            }
            xr[decode_var(fvars[jb + j])] = v;
          }
        }
        if (i0 < npiv) {
          double acc = 0.0;
#pragma unroll
          for (int j = 0; j < SB; j++)
            if (j < bw) acc = __fma_rn((double)a[j], V[jb + j], acc);
          if (bw > SB) acc = __fma_rn((double)a32, V[jb + SB], acc);
          V[i0] -= acc;
        }
        for (int i = je + tid + NT - 32; i < npiv; i += NT)
          V[i] -= dot_strided(L + i + (size_t)jb * f, (size_t)f, bw,
                              [&](int j) { return V[jb + j]; });
      }
    } else if (nstrip > 0) {
      // G[i] -= L21[i, :] y1: s and acc of this thread's first row in
      // registers, of its other rows behind the pivots' values
      double s0 = 0.0, acc0 = 0.0;
      double* more = V + npiv;
      for (int t = tid + NT; t < nrow; t += NT) {
        more[2 * (t - NT)] = 0.0;
        more[2 * (t - NT) + 1] = 0.0;
      }
      const int i0 = row_of(tid);
      const bool on = tid < nrow && i0 < f;
      for (int b = 0; b < nb; b++) {
        const int jb = m.jb[b], bw = m.jb[b + 1] - jb;
        const T* Li = L + (on ? i0 : npiv) + (size_t)jb * f;
        T a[SB];
#pragma unroll
        for (int j = 0; j < SB; j++) a[j] = on && j < bw ? Li[(size_t)j * f] : T(0);
        const T a32 = on && bw > SB ? Li[(size_t)SB * f] : T(0);
        msg::wait(m.bar + b, phase, d.wait_polls, s_leave, err, kCluWait);
        int left = seg - jb % seg;  // columns to the end of the segment
        auto add = [&](double v, int j, double& s, double& acc, int& rest) {
          acc = __fma_rn(v, V[jb + j], acc);
          if (--rest == 0) {
            s += acc;
            acc = 0.0;
            rest = seg;
          }
        };
        int rest = left;
#pragma unroll
        for (int j = 0; j < SB; j++)
          if (j < bw) add((double)a[j], j, s0, acc0, rest);
        if (bw > SB) add((double)a32, SB, s0, acc0, rest);
        for (int t = tid + NT; t < nrow; t += NT) {
          const int i = row_of(t);
          if (i >= f) break;
          const T* Lt = L + i + (size_t)jb * f;
          double s = more[2 * (t - NT)], acc = more[2 * (t - NT) + 1];
          rest = left;
          for (int j = 0; j < bw; j += 16) {
            T e[16];
#pragma unroll
            for (int u = 0; u < 16; u++) e[u] = j + u < bw ? Lt[(size_t)(j + u) * f] : T(0);
#pragma unroll
            for (int u = 0; u < 16; u++)
              if (j + u < bw) add((double)e[u], j + u, s, acc, rest);
          }
          more[2 * (t - NT)] = s;
          more[2 * (t - NT) + 1] = acc;
        }
      }
      if (npiv % seg != 0) {
        s0 += acc0;
        for (int t = tid + NT; t < nrow; t += NT)
          more[2 * (t - NT)] += more[2 * (t - NT) + 1];
      }
      // (armed again for the next right-hand side; the barrier below comes
      // before CTA 0 sends it)
      __syncthreads();
      for (int b = tid; b < nb; b += NT)
        msg::expect(m.bar + b, 8u * (unsigned)(m.jb[b + 1] - m.jb[b]));
      acc0 = s0;
      cluster.sync();
      const double* V0 = cluster.map_shared_rank(V, 0);
      if (on) G[i0] = V0[i0] - acc0;
      for (int t = tid + NT; t < nrow; t += NT) {
        const int i = row_of(t);
        if (i < f) G[i] = V0[i] - more[2 * (t - NT)];
      }
    }
    if (cr == 0 || nstrip == 0) cluster.sync();
    phase ^= 1u;
    cluster.sync();  // CTA 0's vector has been read
  }
  if (__any_sync(0xffffffffu, *(volatile int*)&s_leave.dead))
    msg::leave(&s_leave, err, kCluWait);
}

template <class T>
__global__ void __launch_bounds__(NT, 1)
k_clu_backward(DevicePlan d, const int* __restrict__ nodes, double* x, int nrhs, int ldx,
               double* ubuf, const long long* uoff, int* err) {
  (void)ubuf;
  (void)uoff;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ double sm[];
  __shared__ int s_nb;
  __shared__ msg::Leave s_leave;
  const int cr = (int)cluster.block_rank();
  const int node = nodes[blockIdx.x / CS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWARP = NT / 32;
  const int f = d.f[node], npiv = d.npiv[node];
  const int* fvars = d.ipool + d.ioff[node];
  const T* L = reinterpret_cast<const T*>(d.fpool) + d.foff[node];
  const int ncr = f - npiv;
  const CluSmem m = clu_smem(sm, f, npiv);
  double* V = m.V;            // CTA 0: pivot values, then the columns' corrections
  double* sx = m.V;           // the other CTAs: contribution rows' final values
  const int nb = clu_setup(m, fvars + 3 * f, npiv, false, &s_nb, s_leave);
  double* cor = V + npiv;
  const bool rows = ncr > 0;
  if (cr == 0 && rows)
    for (int b = tid; b < nb; b += NT)
      msg::expect(m.bar + b, 8u * (unsigned)(m.jb[b] - m.jb[b + 1]));
  cluster.sync();
  pdl_enter();
  unsigned phase = 0;
  for (int rhs = blockIdx.y; rhs < nrhs; rhs += gridDim.y) {
    double* xr = x + (long long)rhs * ldx;
    // t[j] = z[j] - L21[:, j]^T x2 for every pivot column, one warp per column
    // over the other CTAs' warps, the last columns first
    if (cr > 0 && rows) {
      for (int r = tid; r < ncr; r += NT) sx[r] = xr[fvars[npiv + r]];
      __syncthreads();
      int b = 0;
      for (int o = (cr - 1) * NWARP + warp; o < npiv; o += CW * NWARP) {
        const int j = npiv - 1 - o;
        while (m.jb[b + 1] > j) b++;
        const double acc = warp_sum_down(lane_dot(L + (size_t)j * f + npiv, 0, ncr, lane,
                                                  [&](int i) { return sx[i]; }));
        if (lane == 0)
          msg::send(msg::remote(cor + j, 0), msg::remote(m.bar + b, 0), acc);
      }
    }
    if (cr == 0) {
      if (nb > 0) fetch_diag<T>(L, f, m.jb[1], m.jb[0] - m.jb[1], m.diag);
      for (int t = tid; t < npiv; t += NT) V[t] = xr[decode_var(fvars[t])];
      // columns jb + (warp - 1) + 7 u of a block are warp's (1 .. 7); their
      // entries of the first 256 rows below the block are loaded while warp 0
      // solves the block before
      constexpr int NW1 = NWARP - 1, CWP = (SB + 1 + NW1 - 1) / NW1, RW = 8;
      T pre[CWP][RW];
      auto load_pre = [&](int jb, int je) {
#pragma unroll
        for (int u = 0; u < CWP; u++)
#pragma unroll
          for (int r = 0; r < RW; r++) {
            const int j = jb + warp - 1 + NW1 * u, i = je + lane + 32 * r;
            pre[u][r] = j < je && i < npiv ? L[i + (size_t)j * f] : T(0);
          }
      };
      if (warp > 0 && nb > 0) load_pre(m.jb[1], m.jb[0]);
      for (int b = 0; b < nb; b++) {
        const int je = m.jb[b], jb = m.jb[b + 1];
        if (rows) msg::wait(m.bar + b, phase, d.wait_polls, s_leave, err, kCluWait);
        cp_wait();
        __syncthreads();  // the last block's values
        // t[j] -= sum_{je <= i < npiv} L[i, j] t[i] for j in [jb, je)
        if (warp > 0) {
#pragma unroll
          for (int u = 0; u < CWP; u++) {
            const int j = jb + warp - 1 + NW1 * u;
            if (j < je) {
              double acc = 0.0;
#pragma unroll
              for (int r = 0; r < RW; r++) {
                const int i = je + lane + 32 * r;
                if (i < npiv) acc = __fma_rn((double)pre[u][r], V[i], acc);
              }
              for (int i = je + lane + 32 * RW; i < npiv; i += 32)
                acc = __fma_rn((double)L[i + (size_t)j * f], V[i], acc);
              acc = warp_sum_down(acc);
              if (lane == 0) V[j] = (rows ? V[j] - cor[j] : V[j]) - acc;
            }
          }
        }
        __syncthreads();
        if (warp == 0)
          upper_block<T>(reinterpret_cast<const T*>(m.diag + (b & 1) * DB), SB + 1, m.K + jb,
                         je - jb, V + jb, lane);
        else if (b + 1 < nb)
          load_pre(m.jb[b + 2], jb);
        if (b + 1 < nb)
          fetch_diag<T>(L, f, m.jb[b + 2], jb - m.jb[b + 2], m.diag + ((b + 1) & 1) * DB);
      }
      __syncthreads();
      for (int j = tid; j < npiv; j += NT) xr[decode_var(fvars[j])] = V[j];
      // (armed again for the next right-hand side; the barrier below comes
      // before its corrections are sent)
      if (rows)
        for (int b = tid; b < nb; b += NT)
          msg::expect(m.bar + b, 8u * (unsigned)(m.jb[b] - m.jb[b + 1]));
    }
    phase ^= 1u;
    cluster.sync();
  }
  if (__any_sync(0xffffffffu, *(volatile int*)&s_leave.dead))
    msg::leave(&s_leave, err, kCluWait);
}

// ---------------------------------------------------------------------------
// Wide fronts (f * npiv large): one cooperative launch per level solves all
// of the level's wide fronts with every CTA of the GPU.  The front vectors
// live in ubuf (global memory).  Each column block of WB pivots alternates
// a sequential phase (one CTA per front solves the block's diagonal
// triangle in shared memory) with a parallel phase (all CTAs apply the
// block to the rows below it, forward, or to the columns left of it,
// backward), separated by grid-wide barriers.  Values other CTAs wrote
// since the last barrier are read with ld.global.cg (L2), never through
// the non-coherent L1.  Sums run in a fixed order: the result does not
// depend on the grid size.
//
// A step is a chain of latencies, not of bytes: the block's diagonal, its
// triangle on one warp, two barriers and a share of the rows.  So the diagonal
// block comes with 20 loads of a thread in flight, and the next one while the
// others are at the rows; and a row's 128 terms are eight warps' partial sums
// over 32-row strips, which occupy a CTA per strip.  One solve of the 3D SIMP
// 20x10x10 KKT (a root of 3,925 pivots) takes 4.5 ms; 5.9 with the block
// fetched at its turn entry by entry and one thread a row.
constexpr int WB = 128;

__device__ __forceinline__ int block_end_w(const int* kind, int jb, int npiv) {
  int je = jb + WB < npiv ? jb + WB : npiv;
  if (je < npiv && kind[je - 1] == 1) je++;
  return je;
}

__device__ __forceinline__ int block_begin_w(const int* kind, int je) {
  int jb = je - WB > 0 ? je - WB : 0;
  if (jb > 0 && kind[jb] == 2) jb--;  // keep 2x2 pairs together
  return jb;
}

template <class T>
struct WideFront {
  int f, npiv;
  const int* fvars;
  const int* kind;
  const T* L;
  double* G;
};

template <class T>
__device__ __forceinline__ WideFront<T> wide_front(const DevicePlan& d, int node,
                                                double* ubuf,
                                                const long long* uoff,
                                                int rhs) {
  WideFront<T> w;
  w.f = d.f[node];
  w.npiv = d.npiv[node];
  w.fvars = d.ipool + d.ioff[node];
  w.kind = w.fvars + 3 * w.f;
  w.L = reinterpret_cast<const T*>(d.fpool) + d.foff[node];
  w.G = ubuf + uoff[node] + (long long)rhs * w.f;
  return w;
}

// Flattened work distribution: item g of a sequence in which front c owns
// cnt_c consecutive items goes to CTA g mod gridDim.x.  Returns this CTA's
// first item of front c, given the number of items before it.
__device__ __forceinline__ long long first_item(long long base) {
  const long long G = gridDim.x;
  long long r = ((long long)blockIdx.x - base) % G;
  return r < 0 ? r + G : r;
}

// The lower triangle of the diagonal block of columns [jb, jb + bw) and its
// pivot kinds into shared memory.
template <class T>
__device__ __forceinline__ void load_wide_block(const WideFront<T>& w, int jb, int bw,
                                                double* sL, int* sK) {
  constexpr int R = (WB + 32) / 32, C = 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j0 = C * warp; j0 < bw; j0 += C * (NT / 32)) {
    T a[C][R];
#pragma unroll
    for (int q = 0; q < C; q++)
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int j = j0 + q, i = lane + 32 * r;
        a[q][r] = j < bw && i >= j && i < bw ? w.L[jb + i + (size_t)(jb + j) * w.f] : T(0);
      }
#pragma unroll
    for (int q = 0; q < C; q++)
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int j = j0 + q, i = lane + 32 * r;
        if (j < bw && i < bw) sL[i + j * (WB + 1)] = a[q][r];
      }
  }
  for (int t = threadIdx.x; t < bw; t += NT) sK[t] = w.kind[jb + t];
}

template <class T>
__global__ void __launch_bounds__(NT)
k_wide_forward(DevicePlan d, const int* __restrict__ nodes, int count,
               double* x, int nrhs, int ldx, double* ubuf,
               const long long* uoff, int* wst) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ double sm[];
  double* sL = sm;                         // (WB + 1)^2 diagonal block
  double* sv = sm + (WB + 1) * (WB + 1);   // WB + 1 block values
  __shared__ int sK[WB + 1];               // the block's pivot kinds
  __shared__ int s_choff;
  __shared__ double part[NT / 32][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int rhs = 0; rhs < nrhs; rhs++) {
    double* xr = x + (long long)rhs * ldx;
    for (int c = blockIdx.x; c < count; c += gridDim.x) {
      const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
      assemble_front_vector(d, nodes[c], w.G, xr, ubuf, uoff, rhs, &s_choff);
      if (tid == 0) {
        wst[2 * c] = 0;
        wst[2 * c + 1] = 0;
      }
    }
    grid.sync();
    // (a CTA with one front fetches its next block ahead)
    const bool one = count <= (int)gridDim.x;
    bool ahead = false;
    int next = 0;  // where its front's next block begins (backward: ends)
    for (;;) {
      // sequential phase: next diagonal block of every front
      for (int c = blockIdx.x; c < count; c += gridDim.x) {
        const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
        const int jb = __ldcg(wst + 2 * c + 1);
        next = jb;
        if (jb >= w.npiv) {
          if (tid == 0) wst[2 * c] = jb;
          continue;
        }
        const int je = block_end_w(w.kind, jb, w.npiv);
        const int bw = je - jb;
        next = je;
        if (!ahead) load_wide_block(w, jb, bw, sL, sK);
        for (int t = tid; t < bw; t += NT) sv[t] = __ldcg(w.G + jb + t);
        __syncthreads();
        if (warp == 0) warp_lower_solve<(WB + 32) / 32>(sL, WB + 1, sK, bw, sv, lane);
        __syncthreads();
        for (int t = tid; t < bw; t += NT) w.G[jb + t] = sv[t];
        if (tid == 0) {
          wst[2 * c] = jb;
          wst[2 * c + 1] = je;
        }
        __syncthreads();
      }
      auto token = grid.barrier_arrive();
      ahead = false;
      if (one && (int)blockIdx.x < count) {
        const WideFront<T> w = wide_front<T>(d, nodes[blockIdx.x], ubuf, uoff, rhs);
        if (next < w.npiv) {
          load_wide_block(w, next, block_end_w(w.kind, next, w.npiv) - next, sL, sK);
          ahead = true;
        }
      }
      grid.barrier_wait(std::move(token));
      bool any = false;
      for (int c = 0; c < count && !any; c++)
        any = __ldcg(wst + 2 * c) < __ldcg(wst + 2 * c + 1);
      if (!any) break;
      // parallel phase: rows below the block, NT rows per item
      long long base = 0;
      for (int c = 0; c < count; c++) {
        const int jb = __ldcg(wst + 2 * c), je = __ldcg(wst + 2 * c + 1);
        if (jb >= je) continue;
        const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
        const long long items = (w.f - je + 31) / 32;
        const int bw = je - jb;
        const int q = (bw + NT / 32 - 1) / (NT / 32);  // terms of a warp
        const int j0 = min(warp * q, bw), nj = min(q, bw - j0);
        bool staged = false;
        for (long long it = first_item(base); it < items; it += gridDim.x) {
          __syncthreads();
          if (!staged) {
            for (int t = tid; t < bw; t += NT) sv[t] = __ldcg(w.G + jb + t);
            __syncthreads();
            staged = true;
          }
          const int i = je + (int)it * 32 + lane;
          part[warp][lane] =
              i < w.f ? dot_strided(w.L + i + (size_t)(jb + j0) * w.f, (size_t)w.f, nj,
                                    [&](int j) { return sv[j0 + j]; })
                      : 0.0;
          __syncthreads();
          if (warp == 0 && i < w.f) {
            double acc = part[0][lane];
#pragma unroll
            for (int p = 1; p < NT / 32; p++) acc = __dadd_rn(acc, part[p][lane]);
            w.G[i] = __ldcg(w.G + i) - acc;
          }
        }
        base += items;
      }
      grid.sync();
    }
    // D^{-1} and the pivots' forward values
    for (int c = blockIdx.x; c < count; c += gridDim.x) {
      const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
      for (int j = tid; j < w.npiv; j += NT) {
        const int kd = w.kind[j];
        const T* L = w.L;
        const size_t f = w.f;
        if (kd == 0) {
          w.G[j] = __ldcg(w.G + j) / L[j + j * f];
        } else if (kd == 1) {
          const double d11 = L[j + j * f];
          const double d21 = L[j + 1 + j * f];
          const double d22 = L[j + 1 + (j + 1) * f];
          const double inv = inv2x2(d11, d21, d22);
          const double x1 = __ldcg(w.G + j), x2 = __ldcg(w.G + j + 1);
          w.G[j] = piv2_first(inv, d21, d22, x1, x2);
          w.G[j + 1] = piv2_second(inv, d11, d21, x1, x2);
        }
      }
      __syncthreads();
      for (int j = tid; j < w.npiv; j += NT)
        xr[decode_var(w.fvars[j])] = __ldcg(w.G + j);
    }
    grid.sync();
  }
}

template <class T>
__global__ void __launch_bounds__(NT)
k_wide_backward(DevicePlan d, const int* __restrict__ nodes, int count,
                double* x, int nrhs, int ldx, double* ubuf,
                const long long* uoff, int* wst) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ double sm[];
  double* sL = sm;
  double* sv = sm + (WB + 1) * (WB + 1);
  __shared__ int sK[WB + 1];  // the block's pivot kinds
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWARP = NT / 32;
  const long long gwarps = (long long)gridDim.x * NWARP;
  for (int rhs = 0; rhs < nrhs; rhs++) {
    double* xr = x + (long long)rhs * ldx;
    for (int c = blockIdx.x; c < count; c += gridDim.x) {
      const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
      for (int r = tid; r < w.npiv; r += NT) w.G[r] = xr[decode_var(w.fvars[r])];
      for (int r = w.npiv + tid; r < w.f; r += NT) w.G[r] = xr[w.fvars[r]];
      if (tid == 0) {
        wst[2 * c] = w.npiv;
        wst[2 * c + 1] = w.npiv;
      }
    }
    grid.sync();
    // t[j] -= sum_{i >= npiv} L[i, j] t[i]: one warp per pivot column
    {
      long long base = 0;
      for (int c = 0; c < count; c++) {
        const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
        const long long gw = (long long)blockIdx.x * NWARP + warp;
        long long r = (gw - base) % gwarps;
        if (r < 0) r += gwarps;
        for (long long j = r; j < w.npiv; j += gwarps) {
          const double acc = warp_sum_down(lane_dot(w.L + (size_t)j * w.f, w.npiv, w.f,
                                                    lane,
                                                    [&](int i) { return __ldcg(w.G + i); }));
          if (lane == 0) w.G[j] = __ldcg(w.G + j) - acc;
        }
        base += w.npiv;
      }
    }
    grid.sync();
    const bool one = count <= (int)gridDim.x;
    bool ahead = false;
    int next = 0;  // where its front's next block begins (backward: ends)
    for (;;) {
      // sequential phase: the next diagonal block from the end
      for (int c = blockIdx.x; c < count; c += gridDim.x) {
        const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
        const int je = __ldcg(wst + 2 * c);
        next = je;
        if (je <= 0) {
          if (tid == 0) wst[2 * c + 1] = je;
          continue;
        }
        const int jb = block_begin_w(w.kind, je);
        const int bw = je - jb;
        next = jb;
        if (!ahead) load_wide_block(w, jb, bw, sL, sK);
        for (int t = tid; t < bw; t += NT) sv[t] = __ldcg(w.G + jb + t);
        __syncthreads();
        if (warp == 0) warp_upper_solve<(WB + 32) / 32>(sL, WB + 1, sK, bw, sv, lane);
        __syncthreads();
        for (int t = tid; t < bw; t += NT) w.G[jb + t] = sv[t];
        if (tid == 0) {
          wst[2 * c] = jb;
          wst[2 * c + 1] = je;
        }
        __syncthreads();
      }
      auto token = grid.barrier_arrive();
      ahead = false;
      if (one && (int)blockIdx.x < count) {
        const WideFront<T> w = wide_front<T>(d, nodes[blockIdx.x], ubuf, uoff, rhs);
        if (next > 0) {
          const int jb = block_begin_w(w.kind, next);
          load_wide_block(w, jb, next - jb, sL, sK);
          ahead = true;
        }
      }
      grid.barrier_wait(std::move(token));
      bool any = false;
      for (int c = 0; c < count && !any; c++)
        any = __ldcg(wst + 2 * c) < __ldcg(wst + 2 * c + 1);
      if (!any) break;
      // parallel phase: t[j] -= sum_{i in block} L[i, j] t[i] for j < jb,
      // one warp per column
      long long base = 0;
      for (int c = 0; c < count; c++) {
        const int jb = __ldcg(wst + 2 * c), je = __ldcg(wst + 2 * c + 1);
        if (jb >= je) continue;
        const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
        const long long gw = (long long)blockIdx.x * NWARP + warp;
        long long r = (gw - base) % gwarps;
        if (r < 0) r += gwarps;
        for (long long j = r; j < jb; j += gwarps) {
          const double acc = warp_sum_down(lane_dot(w.L + (size_t)j * w.f, jb, je, lane,
                                                    [&](int i) { return __ldcg(w.G + i); }));
          if (lane == 0) w.G[j] = __ldcg(w.G + j) - acc;
        }
        base += jb;
      }
      grid.sync();
    }
    for (int c = blockIdx.x; c < count; c += gridDim.x) {
      const WideFront<T> w = wide_front<T>(d, nodes[c], ubuf, uoff, rhs);
      for (int j = tid; j < w.npiv; j += NT)
        xr[decode_var(w.fvars[j])] = __ldcg(w.G + j);
    }
    grid.sync();
  }
}

}  // namespace

#define SCUDA(call)                                                       \
  do {                                                                    \
    cudaError_t e__ = (call);                                             \
    if (e__ != cudaSuccess) {                                             \
      std::fprintf(stderr, "amigo_b200: %s: %s\n", #call,                 \
                   cudaGetErrorString(e__));                              \
      return -2;                                                          \
    }                                                                     \
  } while (0)

// A launch that may start while the previous kernel of the stream drains
// (programmatic stream serialization; the kernel waits in pdl_enter).
template <class... KArgs, class... Args>
static cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block,
                              size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// One cluster of CS CTAs per front (cudaLaunchKernelEx with a cluster
// dimension).
template <class K>
static int launch_cluster(K kernel, int fronts, int smem, cudaStream_t s,
                          const DevicePlan& d, const int* nodes, double* x,
                          int nrhs, int ldx, double* ubuf, const long long* uoff,
                          int* err) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(fronts * CS, std::max(1, std::min(nrhs, kRhsSlices)));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  SCUDA(cudaLaunchKernelEx(&cfg, kernel, d, nodes, x, nrhs, ldx, ubuf, uoff, err));
  ab::count_launch();
  return 0;
}

// Per level: narrow fronts (one CTA each), cluster fronts (CS CTAs each)
// and wide fronts, from the sizes of the last factorization.
static int build_solve_schedule(LdlHandle& h, cudaStream_t s) {
  const int L = h.d.num_levels, nn = h.d.nn;
  // unchanged front sizes (the usual case between IPM iterations): keep it
  if (h.sv_f == h.h_f && h.sv_npiv == h.h_npiv && !h.sv_narrow_ptr.empty() &&
      h.sv_wide_entries == h.wide_entries && h.sv_cluster_entries == h.cluster_entries &&
      h.sv_precision == h.factor_precision) {
    h.solve_epoch = h.factor_epoch;
    return 0;
  }
  h.solve_plan++;
  std::vector<int>& nodes = h.sv_host;
  nodes.clear();
  nodes.reserve(nn);
  h.sv_narrow_ptr.assign(L + 1, 0);
  h.sv_clu_ptr.assign(L + 1, 0);
  h.sv_wide_ptr.assign(L + 1, 0);
  h.sv_narrow_smem.assign(L, 0);
  h.sv_clu_smem.assign(L, 0);
  h.sv_max_wide = 0;
  // a front's class: narrow (one CTA), cluster (CS CTAs) or wide (the
  // cooperative grid), from f * npiv and, for clusters, the front vector
  // fitting in shared memory
  auto cls = [&](int k) {
    const long long e = (long long)h.h_f[k] * h.h_npiv[k];
    if (e >= h.wide_entries) return 2;
    if (e >= h.cluster_entries) {
      if ((long long)clu_bytes(h.h_f[k], h.h_npiv[k]) <= kMaxDynSmem) return 1;
      // (a vector past a CTA's shared memory: the grid, unless it was asked
      // not to)
      if (h.wide_entries < (1ll << 40)) return 2;
    }
    return 0;
  };
  h.sv_small_cnt.assign(L, 0);
  h.sv_small_smem.assign(L, 0);
  // Shared memory of a launch over `fronts` narrow fronts (size f, pivots p):
  // their vectors, and the pivot columns of those that fit the cap (the others
  // read the factor from global memory).  The cap leaves room for as many CTAs
  // per SM as the launch has fronts for, at most four: with more fronts than
  // that a front's latency is hidden by the others'.
  int sms = 0;
  SCUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h.device));
  auto stage_cap = [&](int fronts) -> long long {
    return fronts > 3 * sms ? 48 * 1024 : fronts > sms ? 96 * 1024 : kMaxDynSmem;
  };
  auto stage_bytes = [&](int k) -> long long {
    return (long long)(h.factor_precision == 32
                           ? staged_bytes<float>(h.h_f[k], h.h_npiv[k])
                           : staged_bytes<double>(h.h_f[k], h.h_npiv[k]));
  };
  auto narrow_smem = [&](const int* list, int count, long long cap) -> int {
    long long sm = 0;
    for (int i = 0; i < count; i++) {
      const long long b = stage_bytes(list[i]);
      sm = std::max(sm, b <= cap ? b : std::min<long long>(8ll * h.h_f[list[i]], kMaxDynSmem));
    }
    return (int)((sm + 15) & ~15ll);
  };
  for (int l = 0; l < L; l++) {
    h.sv_narrow_ptr[l] = (int)nodes.size();
    // narrow fronts: the small ones (kSmallThreads-thread CTAs) first
    for (int pass = 0; pass < 2; pass++)
      for (int q = h.level_ptr[l]; q < h.level_ptr[l + 1]; q++) {
        const int k = h.level_nodes[q];
        if (cls(k) == 0 && (h.h_f[k] <= kSmallRows) == (pass == 0)) {
          nodes.push_back(k);
          if (pass == 0) h.sv_small_cnt[l]++;
        }
      }
    {
      const int* list = nodes.data() + h.sv_narrow_ptr[l];
      const int cnt = (int)nodes.size() - h.sv_narrow_ptr[l];
      const long long cap = stage_cap(cnt);
      h.sv_small_smem[l] = narrow_smem(list, h.sv_small_cnt[l], cap);
      // (the launch covers the small fronts too unless they have their own)
      h.sv_narrow_smem[l] = narrow_smem(list, cnt, cap);
    }
    h.sv_clu_ptr[l] = (int)nodes.size();
    long long cm = 0;
    for (int q = h.level_ptr[l]; q < h.level_ptr[l + 1]; q++) {
      const int k = h.level_nodes[q];
      if (cls(k) == 1) {
        nodes.push_back(k);
        cm = std::max(cm, (long long)clu_bytes(h.h_f[k], h.h_npiv[k]));
      }
    }
    h.sv_clu_smem[l] = (int)cm;
    h.sv_wide_ptr[l] = (int)nodes.size();
    for (int q = h.level_ptr[l]; q < h.level_ptr[l + 1]; q++) {
      const int k = h.level_nodes[q];
      if (cls(k) == 2) nodes.push_back(k);
    }
    h.sv_max_wide = std::max(h.sv_max_wide,
                             (int)nodes.size() - h.sv_wide_ptr[l]);
  }
  h.sv_narrow_ptr[L] = h.sv_clu_ptr[L] = h.sv_wide_ptr[L] = (int)nodes.size();
  if (!h.sv_nodes) {
    SCUDA(cudaMalloc((void**)&h.sv_nodes, std::max(nn, 1) * sizeof(int)));
    SCUDA(cudaMalloc((void**)&h.sv_ctr, (kEpochWord + 1) * sizeof(unsigned)));
    SCUDA(cudaMalloc((void**)&h.sv_err, sizeof(int)));
    SCUDA(cudaMemsetAsync(h.sv_ctr, 0, (kEpochWord + 1) * sizeof(unsigned), s));
    SCUDA(cudaMemsetAsync(h.sv_err, 0, sizeof(int), s));
  }
  if (h.sv_max_wide > h.sv_state_cap) {
    if (h.sv_state) SCUDA(cudaFree(h.sv_state));
    h.sv_state = nullptr;
    h.sv_state_cap = std::max(h.sv_max_wide, 16);
    SCUDA(cudaMalloc((void**)&h.sv_state, 2 * h.sv_state_cap * sizeof(int)));
  }
  // nodes is a member: it outlives the asynchronous copy
  SCUDA(cudaMemcpyAsync(h.sv_nodes, nodes.data(), nodes.size() * sizeof(int),
                        cudaMemcpyHostToDevice, s));
  // the all-narrow levels from the leaves, swept by one work-queue launch
  // each way (worth it from two levels)
  int ql = 0;
  while (ql < L && h.sv_clu_ptr[ql] == h.sv_narrow_ptr[ql + 1]) ql++;
  h.sv_qlevels = ql >= 2 ? ql : 0;
  h.sv_qcount = h.sv_qlevels ? h.sv_narrow_ptr[h.sv_qlevels] : 0;
  h.sv_qsmall = true;
  for (int l = 0; l < h.sv_qlevels; l++)
    if (h.sv_small_cnt[l] != h.sv_clu_ptr[l] - h.sv_narrow_ptr[l]) h.sv_qsmall = false;
  if (h.sv_qcount) {
    const int qc = h.sv_qcount;
    // position of each queued node in the forward order
    std::vector<int> pos(nn, -1);
    for (int i = 0; i < qc; i++) pos[nodes[i]] = i;
    std::vector<int>& bq = h.sv_bq_host;
    std::vector<int>& dep = h.sv_dep_host;
    bq.resize(qc);
    dep.resize(qc);
    h.sv_qsmem = narrow_smem(nodes.data(), qc, stage_cap(qc));
    for (int i = 0; i < qc; i++) {
      const int k = nodes[qc - 1 - i];
      const int par = h.sym.node_parent[k];
      bq[i] = k;
      dep[i] = (par >= 0 && pos[par] >= 0) ? par : -1;
    }
    if (!h.sv_bq) {
      SCUDA(cudaMalloc((void**)&h.sv_bq, std::max(nn, 1) * sizeof(int)));
      SCUDA(cudaMalloc((void**)&h.sv_dep, std::max(nn, 1) * sizeof(int)));
      SCUDA(cudaMalloc((void**)&h.sv_done,
                       2 * kRhsSlices * (size_t)std::max(nn, 1) * sizeof(unsigned)));
      SCUDA(cudaMemsetAsync(h.sv_done, 0,
                            2 * kRhsSlices * (size_t)std::max(nn, 1) * sizeof(unsigned), s));
    }
    SCUDA(cudaMemcpyAsync(h.sv_bq, bq.data(), qc * sizeof(int), cudaMemcpyHostToDevice, s));
    SCUDA(cudaMemcpyAsync(h.sv_dep, dep.data(), qc * sizeof(int), cudaMemcpyHostToDevice, s));
  }
  h.sv_qgrid = 0;
  h.sv_f = h.h_f;
  h.sv_npiv = h.h_npiv;
  h.sv_fwd_grid.clear();
  h.sv_wide_entries = h.wide_entries;
  h.sv_cluster_entries = h.cluster_entries;
  h.sv_precision = h.factor_precision;
  h.solve_epoch = h.factor_epoch;
  return 0;
}

template <class T>
static int launch_solve(LdlHandle& h, double* d_x, int nrhs, int ldx,
                        cudaStream_t s) {
  DevicePlan& d = h.d;
  static bool attr_set = false;
  static int wide_grid = 0;
  const size_t wide_smem = ((WB + 1) * (WB + 1) + WB + 1) * sizeof(double);
  if (!attr_set) {
    SCUDA(cudaFuncSetAttribute(k_solve_forward<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_solve_backward<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_solve_forward<T, kSmallThreads>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_solve_backward<T, kSmallThreads>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_solve_forward_q<T, kSmallThreads>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_solve_backward_q<T, kSmallThreads>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_solve_forward_q<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_solve_backward_q<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_clu_forward<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_clu_backward<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               kMaxDynSmem));
    SCUDA(cudaFuncSetAttribute(k_wide_forward<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)wide_smem));
    SCUDA(cudaFuncSetAttribute(k_wide_backward<T>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)wide_smem));
    int dev = 0, sms = 0, bf = 0, bb = 0;
    SCUDA(cudaGetDevice(&dev));
    SCUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bf, k_wide_forward<T>, NT,
                                                        wide_smem));
    SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bb, k_wide_backward<T>,
                                                        NT, wide_smem));
    wide_grid = sms * std::max(1, std::min(bf, bb));
    attr_set = true;
  }
  if ((int)h.sv_fwd_grid.size() != d.num_levels || h.sv_grid_cap != wide_grid) {
    // Cooperative grids sized to the level's work (a grid-wide barrier
    // costs more the more CTAs it spans): forward, one CTA per 32 rows of
    // the level's wide fronts; backward, one per 8 pivot columns (one warp
    // each); at least one per front, at most what is co-resident.
    h.sv_fwd_grid.assign(d.num_levels, 1);
    h.sv_bwd_grid.assign(d.num_levels, 1);
    for (int l = 0; l < d.num_levels; l++) {
      long long fr = 0, bc = 0;
      const int wc = h.sv_narrow_ptr[l + 1] - h.sv_wide_ptr[l];
      for (int q = h.sv_wide_ptr[l]; q < h.sv_narrow_ptr[l + 1]; q++) {
        const int k = h.sv_host[q];
        fr += (h.h_f[k] + 31) / 32;
        bc += (h.h_npiv[k] + 7) / 8;
      }
      h.sv_fwd_grid[l] = (int)std::min<long long>(wide_grid, std::max<long long>(fr, wc));
      h.sv_bwd_grid[l] = (int)std::min<long long>(wide_grid, std::max<long long>(bc, wc));
      h.sv_fwd_grid[l] = std::max(h.sv_fwd_grid[l], 1);
      h.sv_bwd_grid[l] = std::max(h.sv_bwd_grid[l], 1);
    }
    h.sv_grid_cap = wide_grid;
  }
  int* wst = h.sv_state;
  // AMIGO_B200_TRACE=1: device time of every level's sweeps (diagnostics)
  static const bool trace = std::getenv("AMIGO_B200_TRACE") != nullptr;
  std::vector<cudaEvent_t> ev;
  if (trace) {
    ev.resize(2 * d.num_levels + 2);
    for (auto& e : ev) cudaEventCreate(&e);
  }
  const bool queue = (h.solve_queue & 1) && h.sv_qcount > 0;
  const bool small = (h.solve_queue & 2) != 0;
  // (a queue of fronts of at most 128 rows only: 128-thread CTAs)
  const bool qsmall = queue && h.sv_qsmall;
  const int qth = qsmall ? kSmallThreads : NT;
  const int qsm = h.sv_qsmem;
  const unsigned* ep = h.sv_ctr + kEpochWord;   // this solve's epoch, set on the device
  const int slices = std::max(1, std::min(nrhs, kRhsSlices));
  // (without a programmatic launch of its own it starts after everything before
  // it is done: the launches that follow read the factor ahead of their turn)
  { k_sweep_begin<<<1, 32, 0, s>>>(h.sv_ctr); ab::count_launch(); }
  SCUDA(cudaGetLastError());
  if (queue) {
    if (h.sv_qgrid == 0 || h.sv_qgrid_small != qsmall) {
      // CTAs resident at once, at most one per queued front
      int dev = 0, sms = 0, per = 0;
      SCUDA(cudaGetDevice(&dev));
      SCUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      if (qsmall)
        SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per, k_solve_forward_q<T, kSmallThreads>, kSmallThreads, (size_t)qsm));
      else
        SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_solve_forward_q<T>, NT,
                                                            (size_t)qsm));
      h.sv_qgrid = std::max(1, std::min(h.sv_qcount, sms * std::max(per, 1)));
      h.sv_qgrid_small = qsmall;
    }
    if (qsmall)
      SCUDA(launch_pdl(k_solve_forward_q<T, kSmallThreads>, dim3(h.sv_qgrid, slices), dim3(qth),
                       (size_t)qsm, s, d, (const int*)h.sv_nodes, h.sv_qcount, d_x, nrhs,
                       ldx, h.ubuf, (const long long*)h.uoff, qsm / 8, h.sv_ctr, h.sv_done,
                       ep, h.sv_err));
    else
      SCUDA(launch_pdl(k_solve_forward_q<T>, dim3(h.sv_qgrid, slices), dim3(qth), (size_t)qsm, s, d,
                       (const int*)h.sv_nodes, h.sv_qcount, d_x, nrhs, ldx, h.ubuf,
                       (const long long*)h.uoff, qsm / 8, h.sv_ctr, h.sv_done, ep,
                       h.sv_err));
    ab::count_launch();
  }
  for (int l = queue ? h.sv_qlevels : 0; l < d.num_levels; l++) {
    if (trace) cudaEventRecord(ev[l], s);
    int b = h.sv_narrow_ptr[l], cnt = h.sv_clu_ptr[l] - b;
    if (small && h.sv_small_cnt[l]) {
      const int sc = h.sv_small_cnt[l];
      SCUDA(launch_pdl(k_solve_forward<T, kSmallThreads>, dim3(sc, slices), dim3(kSmallThreads),
                       (size_t)h.sv_small_smem[l], s, d, (const int*)(h.sv_nodes + b), d_x,
                       nrhs, ldx, h.ubuf, (const long long*)h.uoff, h.sv_small_smem[l] / 8));
      ab::count_launch();
      b += sc;
      cnt -= sc;
    }
    if (cnt) {
      SCUDA(launch_pdl(k_solve_forward<T>, dim3(cnt, slices), dim3(NT), (size_t)h.sv_narrow_smem[l],
                       s, d, h.sv_nodes + b, d_x, nrhs, ldx, h.ubuf, h.uoff,
                       h.sv_narrow_smem[l] / 8));
      ab::count_launch();
    }
    const int cb = h.sv_clu_ptr[l], ccnt = h.sv_wide_ptr[l] - cb;
    if (ccnt) {
      int rc = launch_cluster(k_clu_forward<T>, ccnt, h.sv_clu_smem[l], s, d,
                              h.sv_nodes + cb, d_x, nrhs, ldx, h.ubuf, h.uoff, h.sv_err);
      if (rc) return rc;
    }
    const int wb = h.sv_wide_ptr[l], wc = h.sv_narrow_ptr[l + 1] - wb;
    if (wc) {
      const int* wn = h.sv_nodes + wb;
      double* ub = h.ubuf;
      const long long* uo = h.uoff;
      void* args[] = {(void*)&d, (void*)&wn, (void*)&wc, (void*)&d_x,
                      (void*)&nrhs, (void*)&ldx, (void*)&ub, (void*)&uo,
                      (void*)&wst};
      SCUDA(cudaLaunchCooperativeKernel((const void*)k_wide_forward<T>,
                                        dim3(h.sv_fwd_grid[l]), dim3(NT), args,
                                        wide_smem, s));
      ab::count_launch();
    }
  }
  if (trace) cudaEventRecord(ev[d.num_levels], s);
  for (int l = d.num_levels - 1; l >= (queue ? h.sv_qlevels : 0); l--) {
    if (trace) cudaEventRecord(ev[d.num_levels + 1 + (d.num_levels - 1 - l)], s);
    int b = h.sv_narrow_ptr[l], cnt = h.sv_clu_ptr[l] - b;
    if (small && h.sv_small_cnt[l]) {
      const int sc = h.sv_small_cnt[l];
      SCUDA(launch_pdl(k_solve_backward<T, kSmallThreads>, dim3(sc, slices), dim3(kSmallThreads),
                       (size_t)h.sv_small_smem[l], s, d, (const int*)(h.sv_nodes + b), d_x,
                       nrhs, ldx, h.ubuf, (const long long*)h.uoff, h.sv_small_smem[l] / 8));
      ab::count_launch();
      b += sc;
      cnt -= sc;
    }
    if (cnt) {
      SCUDA(launch_pdl(k_solve_backward<T>, dim3(cnt, slices), dim3(NT), (size_t)h.sv_narrow_smem[l],
                       s, d, h.sv_nodes + b, d_x, nrhs, ldx, h.ubuf, h.uoff,
                       h.sv_narrow_smem[l] / 8));
      ab::count_launch();
    }
    const int cb = h.sv_clu_ptr[l], ccnt = h.sv_wide_ptr[l] - cb;
    if (ccnt) {
      int rc = launch_cluster(k_clu_backward<T>, ccnt, h.sv_clu_smem[l], s, d,
                              h.sv_nodes + cb, d_x, nrhs, ldx, h.ubuf, h.uoff, h.sv_err);
      if (rc) return rc;
    }
    const int wb = h.sv_wide_ptr[l], wc = h.sv_narrow_ptr[l + 1] - wb;
    if (wc) {
      const int* wn = h.sv_nodes + wb;
      double* ub = h.ubuf;
      const long long* uo = h.uoff;
      void* args[] = {(void*)&d, (void*)&wn, (void*)&wc, (void*)&d_x,
                      (void*)&nrhs, (void*)&ldx, (void*)&ub, (void*)&uo,
                      (void*)&wst};
      SCUDA(cudaLaunchCooperativeKernel((const void*)k_wide_backward<T>,
                                        dim3(h.sv_bwd_grid[l]), dim3(NT), args,
                                        wide_smem, s));
      ab::count_launch();
    }
  }
  if (queue) {
    if (qsmall)
      SCUDA(launch_pdl(k_solve_backward_q<T, kSmallThreads>, dim3(h.sv_qgrid, slices), dim3(qth),
                       (size_t)qsm, s, d, (const int*)h.sv_bq, (const int*)h.sv_dep,
                       h.sv_qcount, d_x, nrhs, ldx, h.ubuf, (const long long*)h.uoff,
                       qsm / 8, h.sv_ctr + kRhsSlices, h.sv_done + (size_t)kRhsSlices * d.nn, ep, h.sv_err));
    else
      SCUDA(launch_pdl(k_solve_backward_q<T>, dim3(h.sv_qgrid, slices), dim3(qth), (size_t)qsm, s, d,
                       (const int*)h.sv_bq, (const int*)h.sv_dep, h.sv_qcount, d_x, nrhs,
                       ldx, h.ubuf, (const long long*)h.uoff, qsm / 8, h.sv_ctr + kRhsSlices,
                       h.sv_done + (size_t)kRhsSlices * d.nn, ep, h.sv_err));
    ab::count_launch();
  }
  if (trace && queue) {
    // the queued levels ran as one launch each way: no per-level times
    for (int l = 0; l < h.sv_qlevels; l++) {
      cudaEventRecord(ev[l], s);
      cudaEventRecord(ev[d.num_levels + 1 + (d.num_levels - 1 - l)], s);
    }
  }
  if (trace) {
    const int L = d.num_levels;
    cudaEventRecord(ev[2 * L + 1], s);
    cudaEventSynchronize(ev[2 * L + 1]);
    float tf = 0.f, tb = 0.f;
    for (int l = 0; l < L; l++) {
      float a = 0.f, b = 0.f;
      cudaEventElapsedTime(&a, ev[l], ev[l + 1]);
      const int bi = L + 1 + (L - 1 - l);
      cudaEventElapsedTime(&b, ev[bi], ev[bi + 1]);
      tf += a;
      tb += b;
      int fm = 0;
      for (int q = h.level_ptr[l]; q < h.level_ptr[l + 1]; q++)
        fm = std::max(fm, h.h_f[h.level_nodes[q]]);
      std::fprintf(stderr,
                   "solve level %d: narrow %d cluster %d wide %d max f %d  fwd %.3f ms  "
                   "bwd %.3f ms\n",
                   l, h.sv_clu_ptr[l] - h.sv_narrow_ptr[l], h.sv_wide_ptr[l] - h.sv_clu_ptr[l],
                   h.sv_narrow_ptr[l + 1] - h.sv_wide_ptr[l], fm, a, b);
    }
    std::fprintf(stderr, "solve total: fwd %.3f ms, bwd %.3f ms\n", tf, tb);
    for (auto& e : ev) cudaEventDestroy(e);
  }
  SCUDA(cudaGetLastError());
  return 0;
}

int solve_numeric(LdlHandle& h, double* d_x, int nrhs, int ldx,
                  cudaStream_t s) {
  DevicePlan& d = h.d;
  const int nn = d.nn;
  if (h.uoff_nrhs != nrhs ||
      (h.solve_epoch != h.factor_epoch && h.sv_f != h.h_f)) {
    // offsets of the update vectors (front sizes change with the delayed
    // pivots of each factorization)
    h.solve_plan++;
    h.h_uoff.resize(nn);
    long long tot = 0;
    for (int k = 0; k < nn; k++) {
      h.h_uoff[k] = tot;
      tot += (long long)h.h_f[k] * nrhs;
    }
    if (tot + 8 > h.ubuf_cap) {
      if (h.ubuf) SCUDA(cudaFree(h.ubuf));
      h.ubuf = nullptr;
      h.ubuf_cap = tot + 8;
      SCUDA(cudaMalloc((void**)&h.ubuf, (size_t)h.ubuf_cap * sizeof(double)));
    }
    SCUDA(cudaMemcpyAsync(h.uoff, h.h_uoff.data(), nn * sizeof(long long),
                          cudaMemcpyHostToDevice, s));
    h.uoff_nrhs = nrhs;
  }
  if (h.solve_epoch != h.factor_epoch) {
    int rc = build_solve_schedule(h, s);
    if (rc) return rc;
  }
  return h.factor_precision == 32 ? launch_solve<float>(h, d_x, nrhs, ldx, s)
                                   : launch_solve<double>(h, d_x, nrhs, ldx, s);
}

}  // namespace ab
