// Solves of one front by one CTA with the front's pivot columns in shared
// memory.  Included by ldl_solve.cu inside its namespace (forward_front and
// backward_front there, which read the factor from global memory, are the
// general form; the arithmetic and its order are the same, so are the bits).
//
// A sweep is a chain of dependent fronts (59 of them for a cart-pole KKT of
// 400 intervals), and a front a chain of dependent steps, so what counts is the
// time from a front's inputs being ready to its results being visible.
// Everything that does not depend on another front -- the factor, the front's
// right-hand side, the index maps -- is fetched before the wait for the
// children (or the parent); after it a step reads shared memory and registers
// only: one warp solves a 32-column diagonal block with its rows' factor
// entries in registers (a broadcast and a multiply-add per column), then every
// thread applies the block to its rows.  One solve: 512 cart-pole KKTs 3.19 ->
// 0.94 ms, one of 100 intervals 0.54 -> 0.20, 24 of FP32 fronts 1.10 -> 0.35.
// Fronts whose pivot columns do not fit the launch's shared memory take the
// general form.

// The pivot kinds of a block as bit masks: first and second column of a pair.
struct BlockKinds {
  unsigned first, second;
};
__device__ __forceinline__ BlockKinds block_kinds(const unsigned char* K, int bw, int lane) {
  const int kd = lane < bw ? K[lane] : 0;
  return BlockKinds{__ballot_sync(0xffffffffu, kd == 1), __ballot_sync(0xffffffffu, kd == 2)};
}

// One warp solves the unit lower triangle of a diagonal block (bw <= 33 rows;
// 33 only when the last two columns are a pair) in place on V[0:bw]; lane i
// holds row i.  Operations and order of warp_lower_solve.
template <class T>
__device__ __forceinline__ void lower_block(const T* L, int lds, const unsigned char* K,
                                            int bw, double* V, int lane) {
  const unsigned FULL = 0xffffffffu;
  const BlockKinds kd = block_kinds(K, min(bw, 32), lane);
  // (columns past the block have zero entries: their steps change nothing)
  T l[32];
  const int last = min(bw, 32) - 1, row = lane < bw ? lane : 0;
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const T a = L[row + min(j, last) * lds];
    l[j] = row > j ? a : T(0);
  }
  double v = lane < bw ? V[lane] : 0.0;
  double part = 0.0;  // the first column's product of a pair
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const double t = __fma_rn((double)l[j], __shfl_sync(FULL, v, j), part);
    const bool first = kd.first >> j & 1u;
    const double nv = __dsub_rn(v, t);
    part = first ? t : 0.0;
    v = row > (first ? 32 : j) ? nv : v;
  }
  if (lane < bw) V[lane] = v;
  if (bw == 33) {
    // the second column of the last pair: columns 0 .. 30 (31 is its partner)
    double w = V[32];
    const double own = lane < 31 ? __dmul_rn((double)L[32 + lane * lds], v) : 0.0;
    const double pre = __shfl_up_sync(FULL, own, 1);
    const double t = kd.second >> lane & 1u
                         ? __fma_rn((double)L[32 + lane * lds], v, pre) : own;
    for (int j = 0; j < 31; j++) {
      const double tj = __shfl_sync(FULL, t, j);
      if (!(kd.first >> j & 1u)) w = __dsub_rn(w, tj);
    }
    if (lane == 0) V[32] = w;
  }
}

// One warp solves the unit upper triangle L^T of a diagonal block (bw <= 33; 33
// only when the first two columns are a pair) in place on V[0:bw], from the
// last pivot backwards; lane i holds row i (bw 33: row i + 1).  Operations and
// order of warp_upper_solve.
template <class T>
__device__ __forceinline__ void upper_block(const T* L, int lds, const unsigned char* K,
                                            int bw, double* V, int lane) {
  const unsigned FULL = 0xffffffffu;
  const int off = bw == 33 ? 1 : 0, nb = bw - off;
  const BlockKinds kd = block_kinds(K + off, nb, lane);
  const int last = nb - 1, row = min(lane, last);
  const T* Lr = L + (size_t)(row + off) * lds + off;  // the lane's column of L
  T l[32];
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const T a = Lr[min(j, last)];
    l[j] = row < j && j < nb ? a : T(0);
  }
  double v = lane < nb ? V[lane + off] : 0.0;
  double part = 0.0;  // the second column's product of a pair
#pragma unroll
  for (int j = 31; j >= 0; j--) {
    const double t = __fma_rn((double)l[j], __shfl_sync(FULL, v, j), part);
    // (the pair's second column subtracts with its first: rows above both)
    const bool second = kd.second >> j & 1u;
    const double nv = __dsub_rn(v, t);
    part = second ? t : 0.0;
    v = row < (second ? -1 : j) ? nv : v;
  }
  if (lane < nb) V[lane + off] = v;
  if (off) {
    // row 0, the first column of the pair (0, 1): columns 32 .. 2
    double w = V[0];
    const double own = lane > 0 ? __dmul_rn((double)L[lane + 1], v) : 0.0;
    const double nxt = __shfl_down_sync(FULL, own, 1);
    const double t = kd.first >> lane & 1u
                         ? __fma_rn((double)L[lane + 1], v, nxt) : own;
    for (int j = 31; j >= 1; j--) {
      const double tj = __shfl_sync(FULL, t, j);
      if (!(kd.second >> j & 1u)) w = __dsub_rn(w, tj);
    }
    if (lane == 0) V[0] = w;
  }
}

// Copy of 4 or 8 bytes to shared memory, in flight until cp_wait.
template <class T>
__device__ __forceinline__ void cp_async_el(T* dst, const T* src) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(a), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(a), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// Shared memory of a staged front: V, the positions of the children's rows
// (forward), the pivot kinds and the pivot columns, the latter with an odd
// leading dimension (rows and columns both fall on distinct banks).
__host__ __device__ __forceinline__ size_t staged_head(int f, int npiv) {
  return (((size_t)f * 8 + (size_t)2 * f * 4 + (size_t)npiv) + 15) & ~(size_t)15;
}
template <class T>
__host__ __device__ __forceinline__ size_t staged_bytes(int f, int npiv) {
  return staged_head(f, npiv) + (size_t)npiv * (f | 1) * sizeof(T);
}

// Lower part of the pivot columns and the pivot kinds to shared memory.
template <class T, int NTH>
__device__ __forceinline__ void stage_columns(const T* L, int f, int npiv, T* Ls, int lds,
                                              const int* kind, unsigned char* K) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = warp; j < npiv; j += NTH / 32)
    for (int r = j + lane; r < f; r += 32)
      cp_async_el(Ls + r + (size_t)j * lds, L + r + (size_t)j * f);
  for (int j = threadIdx.x; j < npiv; j += NTH) K[j] = (unsigned char)kind[j];
}

// Forward solve of one front; after `wait` (a child a thread) the children are
// done.
template <class T, int NTH, class Wait>
__device__ void forward_staged(const DevicePlan& d, int node, double* x, int nrhs, int ldx,
                               double* ubuf, const long long* uoff, char* smem, Wait wait) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f = d.f[node], npiv = d.npiv[node];
  const int ns = d.ns[node], ndin = d.ndin[node], fs = ns + ndin;
  const int* fvars = d.ipool + d.ioff[node];
  const int* fsinv = fvars + 2 * f;
  const int q0 = d.kid_ptr[node], q1 = d.kid_ptr[node + 1];
  double* V = reinterpret_cast<double*>(smem);
  int* P = reinterpret_cast<int*>(V + f);
  unsigned char* K = reinterpret_cast<unsigned char*>(P + 2 * f);
  T* Ls = reinterpret_cast<T*>(smem + staged_head(f, npiv));
  const int lds = f | 1;
  stage_columns<T, NTH>(reinterpret_cast<const T*>(d.fpool) + d.foff[node], f, npiv, Ls, lds,
                        fvars + 3 * f, K);
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
  // positions of the first children's rows (as many as fit)
  int held = 0;
  for (int q = q0, choff = ns, at = 0; q < q1; q++) {
    const int c = d.kids[q], ndc = d.ndel[c], cc = d.f[c] - d.npiv[c];
    if (at + cc > 2 * f) break;
    for (int a = tid; a < cc; a += NTH) P[at + a] = position(c, ndc, choff, a);
    at += cc;
    choff += ndc;
    held = q + 1 - q0;
  }
  const int vb = d.var_ptr[node];
  bool waited = false;
  for (int rhs = blockIdx.y; rhs < nrhs; rhs += gridDim.y) {
    double* G = ubuf + uoff[node] + (long long)rhs * f;
    double* xr = x + (long long)rhs * ldx;
    for (int r = tid; r < f; r += NTH) V[r] = 0.0;
    __syncthreads();
    for (int r = tid; r < ns; r += NTH) V[fsinv[r]] = xr[d.vars[vb + r]];
    if (!waited) {
      cp_wait();
      wait();
      waited = true;
    }
    __syncthreads();
    for (int q = q0, choff = ns, at = 0; q < q1; q++) {
      const int c = d.kids[q], ndc = d.ndel[c], npc = d.npiv[c], cc = d.f[c] - npc;
      const double* uc = ubuf + uoff[c] + (long long)rhs * d.f[c] + npc;
      const bool in_p = q - q0 < held;
      for (int a = tid; a < cc; a += NTH)
        // (from L2: written by another CTA of a queue sweep)
        V[in_p ? P[at + a] : position(c, ndc, choff, a)] += __ldcg(uc + a);
      __syncthreads();
      at += cc;
      choff += ndc;
    }
    for (int jb = 0; jb < npiv;) {
      int je = min(jb + SB, npiv);
      if (je < npiv && K[je - 1] == 1) je++;
      const int bw = je - jb;
      if (warp == 0) lower_block<T>(Ls + jb + (size_t)jb * lds, lds, K + jb, bw, V + jb, lane);
      __syncthreads();
      for (int i = je + tid; i < f; i += NTH) {
        const T* Li = Ls + i + (size_t)jb * lds;
        double acc = 0.0;
        int j = 0;
        for (; j + 8 <= bw; j += 8)
#pragma unroll
          for (int u = 0; u < 8; u++)
            acc = __fma_rn((double)Li[(size_t)(j + u) * lds], V[jb + j + u], acc);
        for (; j < bw; j++) acc = __fma_rn((double)Li[(size_t)j * lds], V[jb + j], acc);
        V[i] -= acc;
      }
      __syncthreads();
      jb = je;
    }
    // the update vector first (the parent waits for it), then D^{-1} and the
    // pivots' forward values
    for (int r = npiv + tid; r < f; r += NTH) G[r] = V[r];
    for (int j = tid; j < npiv; j += NTH) {
      const T* Lj = Ls + j + (size_t)j * lds;
      const int kd = K[j];
      double v;
      if (kd == 0) {
        v = V[j] / (double)Lj[0];
      } else {
        const T* Lf = kd == 1 ? Lj : Lj - lds - 1;  // the pair's first diagonal
        const double d11 = Lf[0], d21 = Lf[1], d22 = Lf[lds + 1];
        const double inv = inv2x2(d11, d21, d22);
        v = kd == 1 ? piv2_first(inv, d21, d22, V[j], V[j + 1])
                    : piv2_second(inv, d11, d21, V[j - 1], V[j]);
      }
      xr[decode_var(fvars[j])] = v;
    }
    __syncthreads();
  }
}

// Backward solve of one front; after `wait` (thread 0) the parent is done.
template <class T, int NTH, class Wait>
__device__ void backward_staged(const DevicePlan& d, int node, double* x, int nrhs, int ldx,
                                char* smem, Wait wait) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NWARP = NTH / 32;
  const int f = d.f[node], npiv = d.npiv[node];
  const int* fvars = d.ipool + d.ioff[node];
  double* V = reinterpret_cast<double*>(smem);
  int* P = reinterpret_cast<int*>(V + f);
  unsigned char* K = reinterpret_cast<unsigned char*>(P + 2 * f);
  T* Ls = reinterpret_cast<T*>(smem + staged_head(f, npiv));
  const int lds = f | 1;
  stage_columns<T, NTH>(reinterpret_cast<const T*>(d.fpool) + d.foff[node], f, npiv, Ls, lds,
                        fvars + 3 * f, K);
  for (int r = tid; r < f; r += NTH) P[r] = r < npiv ? decode_var(fvars[r]) : fvars[r];
  bool waited = false;
  for (int rhs = blockIdx.y; rhs < nrhs; rhs += gridDim.y) {
    double* xr = x + (long long)rhs * ldx;
    // pivots: their forward values; the other rows: final values of the
    // ancestors (from L2: another CTA of the same sweep may have written them)
    for (int r = tid; r < npiv; r += NTH) V[r] = xr[P[r]];
    if (!waited) {
      cp_wait();
      wait();
      waited = true;
      __syncthreads();  // the wait of one thread, and P, for every thread
    }
    for (int r = npiv + tid; r < f; r += NTH) V[r] = __ldcg(xr + P[r]);
    __syncthreads();
    for (int je = npiv; je > 0;) {
      int jb = max(je - SB, 0);
      if (jb > 0 && K[jb] == 2) jb--;  // keep 2x2 pairs together
      // t[j] -= sum_{i >= je} L[i, j] t[i]: four columns a warp, lanes over rows
      for (int j0 = jb + 4 * warp; j0 < je; j0 += 4 * NWARP) {
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        const T* Lj = Ls + (size_t)j0 * lds;
        for (int i = je + lane; i < f; i += 32) {
          const double v = V[i];
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (j0 + u < je) a[u] = __fma_rn((double)Lj[i + (size_t)u * lds], v, a[u]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int u = 0; u < 4; u++) a[u] += __shfl_down_sync(0xffffffffu, a[u], o);
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (lane == 0 && j0 + u < je) V[j0 + u] -= a[u];
      }
      __syncthreads();
      if (warp == 0)
        upper_block<T>(Ls + jb + (size_t)jb * lds, lds, K + jb, je - jb, V + jb, lane);
      __syncthreads();
      je = jb;
    }
    for (int j = tid; j < npiv; j += NTH) xr[P[j]] = V[j];
    __syncthreads();
  }
}
