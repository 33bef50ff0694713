// Element kernels of the SIMP full-space compliance models (2D bilinear
// quads and 3D trilinear hexahedra): gradient of the Lagrangian and its
// Hessian scattered into the CSR KKT pattern.
//
// These replace, for these models, the reference's generated component code
// driven by OptimizationProblem::gradient / hessian
// (include/optimization_problem.h:742-818) and the CUDA atomic scatter
// kernels (include/cuda/component_group_backend.cuh:37-120).  One block per
// element instance: its threads gather the element's variables (coalesced
// from the element's index row), warps 0 and 1 form the rows of K0 u and
// K0 lam, a lane of warp 2 the element scalars, then every thread adds its few
// entries of the element's KKT block at precomputed CSR positions.  Elements
// are processed one colour at a time (no two elements of a colour share a
// node), so the scatter needs no atomics and the result is deterministic.
//
// A colour has at most a few thousand elements, and what one costs is a chain
// of dependent loads (indices, variables, positions, entries), not bandwidth:
// with one warp an element the chain ran once per 32 entries, 98 times for a
// hexahedron.  With a block an element every thread issues its loads at once,
// entries that stay zero (u-u, lam-lam) are not visited, and a colour's blocks
// start while the colour before them runs (programmatic stream serialization):
// everything up to the read of the values depends on x and the model alone.
// Gradient and Hessian of the 3D 24x12x12 model (3,456 elements): 1,027 us
// with one warp an element, 99 so.
#include <cuda_runtime.h>

#include <cmath>

#include "../../include/amigo_b200.h"
#include "launch_count.h"

namespace ab {
namespace {

// Fields shared by ab_simp2d and ab_simp3d.
struct SimpView {
  int n, nnz, nelems, nnodes;
  int u0, rt0, re0, s_index, lam0, mu0, nu_index;
  int ncolors;
  int color_ptr[9];
  const int* color_elems;
  const int* ev;
  const int* fv;
  const int* epos;
  const int* fpos;
  const int* vpos;
  const int* spos;
  const int* fixed;
  const int* fixed_zero_pos;
  const int* fixed_diag_pos;
  const int* load_idx;
  const double* load_val;
  const double* K0;
  const double* A;
  int nfixed, nfixed_zero, nload;
  double Bq, vcoef, volfrac, E0, Emin, penalty;
};

template <class M>
SimpView view(const M* m, int ncolors) {
  SimpView v;
  v.n = m->n; v.nnz = m->nnz; v.nelems = m->nelems; v.nnodes = m->nnodes;
  v.u0 = m->u0; v.rt0 = m->rt0; v.re0 = m->re0; v.s_index = m->s_index;
  v.lam0 = m->lam0; v.mu0 = m->mu0; v.nu_index = m->nu_index;
  v.ncolors = ncolors;
  for (int c = 0; c < 9; c++) v.color_ptr[c] = c <= ncolors ? m->color_ptr[c] : 0;
  v.color_elems = m->color_elems; v.ev = m->ev; v.fv = m->fv;
  v.epos = m->epos; v.fpos = m->fpos; v.vpos = m->vpos; v.spos = m->spos;
  v.fixed = m->fixed; v.fixed_zero_pos = m->fixed_zero_pos;
  v.fixed_diag_pos = m->fixed_diag_pos; v.load_idx = m->load_idx;
  v.load_val = m->load_val; v.K0 = m->K0; v.A = m->A;
  v.nfixed = m->nfixed; v.nfixed_zero = m->nfixed_zero; v.nload = m->nload;
  v.Bq = m->Bq; v.vcoef = m->vcoef; v.volfrac = m->volfrac; v.E0 = m->E0;
  v.Emin = m->Emin; v.penalty = m->penalty;
  return v;
}

// Element sizes: NV nodes, ND displacement dofs, NE = |ev row|, NF = |fv row|.
// NH entries of the elasticity block and NP of the filter block are non-zero.
template <int DIM>
struct Dims {
  static constexpr int NV = 1 << DIM;
  static constexpr int ND = DIM * NV;
  static constexpr int NE = 2 * ND + NV;
  static constexpr int NF = 2 * NV + 1;
  static constexpr int NH = 2 * ND * (NV + ND) + NV * NE;
  static constexpr int NP = 2 * NV * NV + 2 * NV;
  static constexpr int THREADS = DIM == 3 ? 256 : 128;
  static_assert(THREADS >= NE + 1 + NV && THREADS >= NP && THREADS >= 96, "one pass");
};

// An element's data: its variables v (u | rt | lam), Ku = K0 u, Kl = K0 lam,
// sc = {E, dE, d2E, lam^T K0 u}, and the matrices (rows of K0 on distinct
// banks).
template <int DIM>
struct Slot {
  using D = Dims<DIM>;
  static constexpr int LD = D::ND + 1;
  double K0[D::ND * LD], A[D::NV * D::NV];
  double v[D::NE], Ku[D::ND], Kl[D::ND], sc[4];
};

__device__ __forceinline__ void stiffness(const SimpView& m, double r,
                                          double& E, double& dE,
                                          double& d2E) {
  const double p = m.penalty, dEr = m.E0 - m.Emin;
  const double rp2 = pow(r, p - 2.0);
  E = m.Emin + rp2 * r * r * dEr;
  dE = p * rp2 * r * dEr;
  d2E = p * (p - 1.0) * rp2 * dEr;
}

// Fills the slot for element e; ends with a barrier.
template <int DIM>
__device__ __forceinline__ void element_slot(const SimpView& m, const double* x, int e,
                                             Slot<DIM>& s) {
  using D = Dims<DIM>;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int* ev = m.ev + (size_t)e * D::NE;
  if (tid < D::NE) s.v[tid] = x[ev[tid]];
  for (int t = tid; t < D::ND * D::ND; t += D::THREADS)
    s.K0[t / D::ND * Slot<DIM>::LD + t % D::ND] = m.K0[t];
  if (tid < D::NV * D::NV) s.A[tid] = m.A[tid];
  __syncthreads();
  const double* lam = s.v + D::ND + D::NV;
  if (warp < 2) {
    const double* w = warp == 0 ? s.v : lam;
    if (lane < D::ND) {
      double k = 0.0;
#pragma unroll
      for (int b = 0; b < D::ND; b++) k += s.K0[lane * Slot<DIM>::LD + b] * w[b];
      (warp == 0 ? s.Ku : s.Kl)[lane] = k;
    }
    __syncwarp();
    if (tid == 0) {
      double lku = 0.0;
#pragma unroll
      for (int a = 0; a < D::ND; a++) lku += lam[a] * s.Ku[a];
      s.sc[3] = lku;
    }
  } else if (tid == 64) {
    const double* rt = s.v + D::ND;
    double r = 0.0;
    for (int a = 0; a < D::NV; a++) r += rt[a];
    r *= 1.0 / D::NV;
    stiffness(m, r, s.sc[0], s.sc[1], s.sc[2]);
  }
  __syncthreads();
}

// Before this the kernels read x and the model only, which the work ahead of
// the first colour wrote; after it the values of the colour before are there.
__device__ __forceinline__ void wait_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void let_next_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The first colour's launch has one block more, for the slack's entries.
template <int DIM>
__global__ void __launch_bounds__(Dims<DIM>::THREADS)
k_simp_hessian(SimpView m, const int* __restrict__ elems, int count,
               const double* __restrict__ x, double* __restrict__ vals) {
  using D = Dims<DIM>;
  __shared__ Slot<DIM> s;
  let_next_start();
  const int tid = threadIdx.x;
  if (blockIdx.x == count) {
    if (tid < 2) vals[m.spos[tid]] += -1.0;
    return;
  }
  const int e = elems[blockIdx.x];
  constexpr int R0 = D::ND, L0 = D::ND + D::NV;  // first rt / lam slot
  constexpr int WU = D::NV + D::ND;              // entries of a u or lam row
  constexpr int N = (D::NH + D::THREADS - 1) / D::THREADS;
  // elasticity block: rows u (columns rt, lam), rt (all), lam (columns u, rt)
  auto entry = [&](int t, int& r, int& c) {
    if (t < D::ND * WU) {
      r = t / WU;
      c = R0 + t % WU;
    } else if (t < D::ND * WU + D::NV * D::NE) {
      r = R0 + (t - D::ND * WU) / D::NE;
      c = (t - D::ND * WU) % D::NE;
    } else {
      t -= D::ND * WU + D::NV * D::NE;
      r = L0 + t / WU;
      c = t % WU;
    }
  };
  const int* ep = m.epos + (size_t)e * D::NE * D::NE;
  int pos[N];
#pragma unroll
  for (int i = 0; i < N; i++) {
    const int t = tid + i * D::THREADS;
    int r = 0, c = 0;
    if (t < D::NH) entry(t, r, c);
    pos[i] = t < D::NH ? ep[r * D::NE + c] : -1;
  }
  // Helmholtz filter block [rt(NV) | re | mu(NV)] (linear: Jacobian only):
  // mu-rt, rt-mu, mu-re, re-mu
  constexpr int V = D::NV;
  int fpos = -1, fa = -1;
  if (tid < D::NP) {
    int r, c;
    if (tid < V * V) {
      r = V + 1 + tid / V;
      c = tid % V;
      fa = (r - V - 1) * V + c;
    } else if (tid < 2 * V * V) {
      r = (tid - V * V) / V;
      c = V + 1 + tid % V;
      fa = (c - V - 1) * V + r;
    } else if (tid < 2 * V * V + V) {
      r = V + 1 + tid - 2 * V * V;
      c = V;
    } else {
      r = V;
      c = V + 1 + tid - 2 * V * V - V;
    }
    fpos = m.fpos[(size_t)e * D::NF * D::NF + r * D::NF + c];
  }
  const int vpos = tid < 2 ? m.vpos[2 * e + tid] : -1;
  element_slot<DIM>(m, x, e, s);
  const double E = s.sc[0];
  const double q1 = s.sc[1] * (1.0 / D::NV);
  const double q2 = s.sc[2] * s.sc[3] * (1.0 / (D::NV * D::NV));
  double val[N];
#pragma unroll
  for (int i = 0; i < N; i++) {
    const int t = tid + i * D::THREADS;
    int r = 0, c = 0;
    if (t < D::NH) entry(t, r, c);
    const bool rr = r >= R0 && r < L0, cr = c >= R0 && c < L0;
    if (rr && cr) {
      val[i] = q2;
    } else if (rr || cr) {
      const int o = rr ? c : r;  // the displacement or multiplier slot
      val[i] = q1 * (o < R0 ? s.Kl[o] : s.Ku[o - L0]);
    } else {
      val[i] = r < R0 ? E * s.K0[r * Slot<DIM>::LD + max(c - L0, 0)]
                      : E * s.K0[(r - L0) * Slot<DIM>::LD + c];
    }
  }
  wait_previous();
  double old[N];
#pragma unroll
  for (int i = 0; i < N; i++) old[i] = pos[i] >= 0 ? vals[pos[i]] : 0.0;
  const double oldf = fpos >= 0 ? vals[fpos] : 0.0;
  const double oldv = vpos >= 0 ? vals[vpos] : 0.0;
#pragma unroll
  for (int i = 0; i < N; i++)
    if (pos[i] >= 0) vals[pos[i]] = __dadd_rn(old[i], val[i]);
  if (fpos >= 0) vals[fpos] = oldf + (fa >= 0 ? s.A[fa] : -m.Bq);
  if (vpos >= 0) vals[vpos] = oldv + m.vcoef;
}

// The volume row v^T re - volfrac - s and the slack column -nu: the rows no
// element adds to.  The sum runs over 256 interleaved partial sums, folded as
// a tree, whatever the block's threads.
template <int BT>
__device__ void volume_rows(const SimpView& m, const double* x, double* g) {
  constexpr int P = 256 / BT;
  __shared__ double part[BT];
  double acc[P];
#pragma unroll
  for (int p = 0; p < P; p++) acc[p] = 0.0;
#pragma unroll 4
  for (int e = threadIdx.x; e < m.nelems; e += 256)
#pragma unroll
    for (int p = 0; p < P; p++)
      if (e + p * BT < m.nelems) acc[p] += x[m.re0 + e + p * BT];
#pragma unroll
  for (int o = P / 2; o > 0; o >>= 1)
#pragma unroll
    for (int p = 0; p < o; p++) acc[p] += acc[p + o];
  part[threadIdx.x] = acc[0];
  __syncthreads();
  for (int o = BT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    g[m.nu_index] += m.vcoef * part[0] - m.volfrac - x[m.s_index];
    g[m.s_index] += -x[m.nu_index];
  }
}

// The first colour's launch has one block more, for the volume rows.
template <int DIM>
__global__ void __launch_bounds__(Dims<DIM>::THREADS)
k_simp_gradient(SimpView m, const int* __restrict__ elems, int count,
                const double* __restrict__ x, double* __restrict__ g) {
  using D = Dims<DIM>;
  __shared__ Slot<DIM> s;
  let_next_start();
  if (blockIdx.x == count) {
    volume_rows<D::THREADS>(m, x, g);
    return;
  }
  const int e = elems[blockIdx.x];
  constexpr int V = D::NV, R0 = D::ND, L0 = D::ND + D::NV;
  const int* ev = m.ev + (size_t)e * D::NE;
  const int* fv = m.fv + (size_t)e * D::NF;
  // rows: ev slots (u | rt | lam), then re, then the V filter multipliers
  const int t = threadIdx.x;
  const bool on = t < D::NE + 1 + V;
  int row = -1;
  if (on) row = t < D::NE ? ev[t] : fv[V + t - D::NE];
  double mu[V];  // the filter multipliers, for the rows that need them
  const bool filt = on && ((t >= R0 && t < L0) || t == D::NE);
#pragma unroll
  for (int k = 0; k < V; k++) mu[k] = filt ? x[fv[V + 1 + k]] : 0.0;
  const double re = on && t > D::NE ? x[fv[V]] : 0.0;
  element_slot<DIM>(m, x, e, s);
  const double* rt = s.v + R0;
  double val = 0.0;
  if (t < R0) {
    val = s.sc[0] * s.Kl[t];
  } else if (t < L0) {
    val = (1.0 / V) * s.sc[1] * s.sc[3];
#pragma unroll
    for (int k = 0; k < V; k++) val += mu[k] * s.A[k * V + t - R0];
  } else if (t < D::NE) {
    val = s.sc[0] * s.Ku[t - L0];
  } else if (t == D::NE) {
    double smu = 0.0;
#pragma unroll
    for (int k = 0; k < V; k++) smu += mu[k];
    val = -m.Bq * smu + m.vcoef * x[m.nu_index];
  } else if (on) {
    const int k = t - D::NE - 1;
    val = -m.Bq * re;
    for (int l = 0; l < V; l++) val += s.A[k * V + l] * rt[l];
  }
  wait_previous();
  if (on) g[row] = __dadd_rn(g[row], val);
}

// Load terms: alpha f^T u, and -f in the equilibrium residual.
__global__ void k_simp_load(SimpView m, double alpha, double* g) {
  wait_previous();
  for (int t = threadIdx.x; t < m.nload; t += blockDim.x) {
    const int i = m.load_idx[t];
    g[m.u0 + i] += alpha * m.load_val[t];
    g[m.lam0 + i] -= m.load_val[t];
  }
}

__global__ void k_set_values(int n, const int* pos, double v, double* vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = i < n ? pos[i] : -1;
  wait_previous();
  if (p >= 0) vals[p] = v;
}

// A launch that may start while the one before it in the stream runs.
template <class... KArgs, class... Args>
void launch(bool overlap, void (*kernel)(KArgs...), int grid, int block, cudaStream_t s,
            Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, args...);
  ab::count_launch();
}

// Only the first colour waits for the work ahead of it in the stream as a
// whole; the others overlap the colour before them.
template <int DIM>
int gradient(const SimpView& m, const double* x, double alpha, double* grad,
             cudaStream_t s) {
  using D = Dims<DIM>;
  cudaMemsetAsync(grad, 0, (size_t)m.n * sizeof(double), s);
  for (int c = 0; c < m.ncolors; c++) {
    const int cnt = m.color_ptr[c + 1] - m.color_ptr[c];
    if (cnt || c == 0)
      launch(c > 0, k_simp_gradient<DIM>, cnt + (c == 0), D::THREADS, s, m,
             m.color_elems + m.color_ptr[c], cnt, x, grad);
  }
  if (m.nload) launch(true, k_simp_load, 1, 256, s, m, alpha, grad);
  // fixed variables: zero their gradient rows
  if (m.nfixed)
    launch(true, k_set_values, (m.nfixed + 255) / 256, 256, s, m.nfixed, m.fixed, 0.0, grad);
  return cudaGetLastError() == cudaSuccess ? AB_OK : AB_ERR_CUDA;
}

template <int DIM>
int hessian(const SimpView& m, const double* x, double* vals, cudaStream_t s) {
  using D = Dims<DIM>;
  cudaMemsetAsync(vals, 0, (size_t)m.nnz * sizeof(double), s);
  for (int c = 0; c < m.ncolors; c++) {
    const int cnt = m.color_ptr[c + 1] - m.color_ptr[c];
    if (cnt || c == 0)
      launch(c > 0, k_simp_hessian<DIM>, cnt + (c == 0), D::THREADS, s, m,
             m.color_elems + m.color_ptr[c], cnt, x, vals);
  }
  if (m.nfixed_zero)
    launch(true, k_set_values, (m.nfixed_zero + 255) / 256, 256, s, m.nfixed_zero,
           m.fixed_zero_pos, 0.0, vals);
  if (m.nfixed)
    launch(true, k_set_values, (m.nfixed + 255) / 256, 256, s, m.nfixed, m.fixed_diag_pos,
           1.0, vals);
  return cudaGetLastError() == cudaSuccess ? AB_OK : AB_ERR_CUDA;
}

}  // namespace
}  // namespace ab

extern "C" {

int ab_simp2d_gradient(const ab_simp2d* m, const double* x, double alpha,
                       double* grad, void* stream) {
  if (!m || !x || !grad) return AB_ERR_ARG;
  return ab::gradient<2>(ab::view(m, 4), x, alpha, grad, (cudaStream_t)stream);
}

int ab_simp2d_hessian(const ab_simp2d* m, const double* x, double alpha,
                      double* vals, void* stream) {
  (void)alpha;  // the objective f^T u is linear: no Hessian term
  if (!m || !x || !vals) return AB_ERR_ARG;
  return ab::hessian<2>(ab::view(m, 4), x, vals, (cudaStream_t)stream);
}

int ab_simp3d_gradient(const ab_simp3d* m, const double* x, double alpha,
                       double* grad, void* stream) {
  if (!m || !x || !grad) return AB_ERR_ARG;
  return ab::gradient<3>(ab::view(m, 8), x, alpha, grad, (cudaStream_t)stream);
}

int ab_simp3d_hessian(const ab_simp3d* m, const double* x, double alpha,
                      double* vals, void* stream) {
  (void)alpha;
  if (!m || !x || !vals) return AB_ERR_ARG;
  return ab::hessian<3>(ab::view(m, 8), x, vals, (cudaStream_t)stream);
}

}  // extern "C"
