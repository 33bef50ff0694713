// Factorization of a small front in shared memory by one CTA: unblocked and
// right-looking, every pivot's rank-1 (2x2: rank-2) update applied to the
// trailing lower triangle at once.  Included by ldl_factor.cu inside its
// namespace; the pivot rule, interchanges and the entries' operations and order
// are those of factor_front_rl, which is the general form (any size, any
// memory).
//
// A front of 68 rows and 63 pivots is a chain of 63 steps, and with 17,000 of
// them in a batch of 512 problems a few hundred fronts share the GPU at a time,
// so both a step's latency and its instructions count.  Per step: every warp
// takes the decision itself from the candidate column's scan (left by the last
// update), keeps the pivot's L column in registers (one row a lane, NCH chunks
// of 32 rows), and applies it to columns of the triangle, lanes over rows; warp 0
// updates the next candidate column alone and folds its scan with warp
// reductions on the entries' bits.  One barrier a step; an interchange adds two.
// The columns are padded to whole chunks and the update runs over whole chunks:
// what it leaves above the diagonal and in the padding is never read, and no
// entry needs a test of its own (with tests: 405 instructions a warp and step,
// and no gain).  A step is bound by its instructions and the chain of decision,
// interchange and update, not by a pipe; 256 threads against 128 and before
// (column scans and folds of the whole CTA, a barrier each), factorization
// time: cart-pole KKT of 100 intervals 0.93 ms (1.11 with 128 threads, 1.20
// before), 512 trajectories at once 5.59 (6.12, 6.68), 24 of them in FP32 1.75
// (2.04, 2.31), 2D SIMP 32x16 2.70 (2.87, 2.97).
constexpr int kSmallChunks = 5;  // rows: 160, past what shared memory holds

struct SmallCtl {
  RowEntry scan[2];  // the next candidate column's scan, by step parity
};

// Leading dimension of a front in shared memory: whole chunks of rows and one
// more (rows and columns on distinct banks).  Its entries are rounded to 16
// bytes; five sections of f ints follow.
__host__ __device__ __forceinline__ int small_ld(int f) { return ((f + 31) & ~31) + 1; }
template <class T>
__host__ __device__ __forceinline__ size_t small_entries(int f) {
  constexpr size_t al = 16 / sizeof(T);
  return ((size_t)f * small_ld(f) + al - 1) / al * al;
}
template <class T>
__host__ __device__ __forceinline__ size_t small_bytes(int f) {
  return small_entries<T>(f) * sizeof(T) + (size_t)5 * f * 4;
}

// Zero, the entries of A, extend-add of the children one after another (a warp
// per column of a child); every entry gets its terms in assemble_front's order.
template <class T, int BT>
__device__ __forceinline__ void small_assemble(const DevicePlan& d, int node, T* F, int ld,
                                               int f, int ns, int ndin,
                                               const double* __restrict__ vals, int* rmap) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  {
    int4* Z = reinterpret_cast<int4*>(F);
    const int nz = (int)(small_entries<T>(f) * sizeof(T) / 16);
    for (int t = tid; t < nz; t += BT) Z[t] = make_int4(0, 0, 0, 0);
  }
  __syncthreads();
  {
    const int a0 = d.amap_ptr[node], a1 = d.amap_ptr[node + 1];
    for (int t0 = a0 + tid; t0 < a1; t0 += 4 * BT) {
      int pos[4];
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int t = t0 + u * BT;
        pos[u] = -1;
        if (t < a1) {
          const int r0 = d.amap_row[t];
          pos[u] = (r0 < ns ? r0 : r0 + ndin) + d.amap_col[t] * ld;
          v[u] = vals[d.amap_pos[t]];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (pos[u] >= 0) F[pos[u]] += T(v[u]);
    }
  }
  __syncthreads();
  const T* pool = reinterpret_cast<const T*>(d.fpool);
  int choff = ns;
  for (int q = d.kid_ptr[node]; q < d.kid_ptr[node + 1]; q++) {
    const int c = d.kids[q];
    const int fc = d.f[c], npc = d.npiv[c], ndc = d.ndel[c];
    const int cc = fc - npc;
    const T* C = pool + d.foff[c];
    const int cb = d.cptr[c];
    for (int a = tid; a < cc; a += BT)
      rmap[a] = child_row_pos(d, cb, ndc, choff, ns, ndin, a);
    __syncthreads();
    for (int b = warp; b < cc; b += BT / 32) {
      const int pb = rmap[b];
      const T* Cb = C + (size_t)(npc + b) * fc + npc;
      for (int a = b + lane; a < cc; a += 32) {
        const int pa = rmap[a];
        F[max(pa, pb) + min(pa, pb) * ld] += Cb[a];
      }
    }
    __syncthreads();
    choff += ndc;
  }
}

// The rows of one lane: lane + 32 i.  l0 (and l1): L entries of the pivot
// column(s) at k; columns c0 .. n - 1 of the triangle updated, column c0 by warp
// 0, which leaves its scan in `scan`.  Returns whether it did (c0 < n).
template <class T, int BT, int NCH, int STEP>
__device__ __forceinline__ bool small_update(T* F, int n, int k, int c0, int nc,
                                             const T (&l0)[NCH], const T (&l1)[NCH],
                                             RowEntry* scan) {
  constexpr int NW = BT / 32, ld = 32 * NCH + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* W0 = F + k * ld;
  const T* W1 = W0 + ld;
  if (c0 >= n) return false;
  if (warp == 0) {
    const T y0 = W0[c0];
    const T y1 = STEP == 2 ? W1[c0] : T(0);
    T* Fc = F + c0 * ld + lane;
    RowEntry e{0u, 0u, kNoPos, 0u, 0u, 0u, 0u, 0u};
    T acc[NCH];
#pragma unroll
    for (int i = 0; i < NCH; i++) acc[i] = Fc[32 * i];
#pragma unroll
    for (int i = 0; i < NCH; i++) {
      acc[i] = fma(-l0[i], y0, acc[i]);
      if (STEP == 2) acc[i] = fma(-l1[i], y1, acc[i]);
      Fc[32 * i] = acc[i];
    }
#pragma unroll
    for (int i = 0; i < NCH; i++) {
      const int r = lane + 32 * i;
      const double a = fabs((double)acc[i]);
      row_argmax(e, a, r, r > c0 && r < nc);
      row_max(e, a, r >= max(nc, c0 + 1) && r < n);
    }
    row_fold(e);
    if (lane == 0) *scan = e;
    return true;
  }
  for (int c = c0 + warp; c < n; c += NW - 1) {
    const T y0 = W0[c];
    const T y1 = STEP == 2 ? W1[c] : T(0);
    T* Fc = F + c * ld + lane;
#pragma unroll
    for (int i = 0; i < NCH; i++)
      if (i == NCH - 1 || c < 32 * (i + 1)) {
        T acc = fma(-l0[i], y0, Fc[32 * i]);
        if (STEP == 2) acc = fma(-l1[i], y1, acc);
        Fc[32 * i] = acc;
      }
  }
  return true;
}

// Factor the fully-summed columns [0, fs) of the n x n front F (lower triangle,
// leading dimension ld); `vars` holds four sections of n ints.  Returns the
// number of pivots.
template <class T, int BT, int NCH>
__device__ int small_factor(T* F, int n, int fs, bool root, int* vars, int* fsperm,
                            double ustab, double pivot_tol, int* status, SmallCtl& sc) {
  constexpr int ld = 32 * NCH + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int k = 0, nc = fs;
  int par = 0;        // parity of the scan slot the next step reads
  bool have = false;  // the update left the scan of column k in slot par
  // the last pivot, whose L column(s) are stored at the next step
  int pk = -1, pstep = 0;
  T l0[NCH], l1[NCH];
  auto store_l = [&]() {
    if (pk < 0) return;
    // (warp 1 the first column, warp 2 the second)
    if (warp == 1 || (pstep == 2 && warp == 2)) {
      T* Fc = F + (pk + warp - 1) * ld;
#pragma unroll
      for (int i = 0; i < NCH; i++) {
        const int r = lane + 32 * i;
        if (r >= pk + pstep) Fc[r] = warp == 1 ? l0[i] : l1[i];
      }
    }
    pk = -1;
  };
  while (k < nc) {
    store_l();
    const T* Fk = F + k * ld;
    RowEntry e;
    if (have) {
      e = sc.scan[par];
    } else {
      // candidate column k: first-argmax over candidates r > k, maximum over
      // the non-candidate rows
      e = RowEntry{0u, 0u, kNoPos, 0u, 0u, 0u, 0u, 0u};
      for (int r = k + 1 + lane; r < n; r += 32) {
        const double a = fabs((double)Fk[r]);
        row_argmax(e, a, r, r < nc);
        row_max(e, a, r >= nc);
      }
      row_fold(e);
    }
    const double wkk = (double)Fk[k];
    const double abswik = row_bits(e.h, e.l), ctail = row_bits(e.th, e.tl);
    const bool tails = e.th > e.h || (e.th == e.h && e.tl > e.l);
    int imax = (int)e.i;
    if (imax >= nc || imax <= k) {
      // no finite candidate entry (all NaN, or no candidates)
      if (k + 1 < nc && tid == 0) atomicOr(status, ST_NAN);
      imax = (k + 1 < n) ? k + 1 : k;
    }
    PivotChoice pc{1, k, false, false};
    if (!plain_pivot(root, wkk, tails ? ctail : abswik, ustab, pivot_tol)) {
      ImaxColumn ic{0.0, 0.0, 0.0};
      if (needs_imax(root, k, nc, wkk, abswik, ctail, ustab, pivot_tol)) {
        RowEntry m{0u, 0u, kNoPos, 0u, 0u, 0u, 0u, 0u};
        for (int r = k + lane; r < n; r += 32)
          row_max(m, fabs((double)F[max(r, imax) + min(r, imax) * ld]), r != imax);
        row_fold_max(m.th, m.tl);
        ic = ImaxColumn{row_bits(m.th, m.tl), (double)F[imax + imax * ld], (double)Fk[imax]};
        // every warp has read column imax, and the last pivot's L columns are
        // stored, before any thread interchanges or updates
        __syncthreads();
      }
      pc = choose_pivot(root, k, nc, wkk, imax, abswik, ctail, ustab, pivot_tol,
                        [&]() { return ic; });
    }
    const int step = pc.step;
    const int from = step == 0 ? k : k + step - 1, to = step == 0 ? nc - 1 : pc.kpiv;
    if (from < to) {
      symm_swap<T, BT>(F, ld, n, vars, fsperm, from, to);
      __syncthreads();
    }
    if (step == 0) {
      // delay candidate k: it moved to the end of the candidate set
      nc -= 1;
      have = false;
      continue;
    }
    const int c0 = k + step;
    if (step == 1) {
      const T d = Fk[k];
      if (!isfinite((double)d) && tid == 0) atomicOr(status, ST_NAN);
      const T dinv = pc.zero ? T(0) : T(1) / d;
      if (tid == 0) vars[3 * n + k] = 0;  // 1x1 pivot
#pragma unroll
      for (int i = 0; i < NCH; i++) l0[i] = Fk[lane + 32 * i] * dinv;
      have = small_update<T, BT, NCH, 1>(F, n, k, c0, nc, l0, l0, &sc.scan[par ^ 1]);
    } else {
      const T* W1 = Fk + ld;
      const T d11 = Fk[k], d21 = Fk[k + 1], d22 = W1[k + 1];
      const T detinv = T(1) / (d11 * d22 - d21 * d21);
      if (!isfinite((double)detinv) && tid == 0) atomicOr(status, ST_NAN);
      const T i00 = d22 * detinv, i10 = -d21 * detinv,
              i01 = -d21 * detinv, i11 = d11 * detinv;
#pragma unroll
      for (int i = 0; i < NCH; i++) {
        const T w0 = Fk[lane + 32 * i], w1 = W1[lane + 32 * i];
        l0[i] = w0 * i00 + w1 * i10;
        l1[i] = w0 * i01 + w1 * i11;
      }
      have = small_update<T, BT, NCH, 2>(F, n, k, c0, nc, l0, l1, &sc.scan[par ^ 1]);
      if (tid == 0) {
        vars[k] = -(vars[k] + 1);
        vars[k + 1] = -(vars[k + 1] + 1);
        vars[3 * n + k] = 1;
        vars[3 * n + k + 1] = 2;
      }
    }
    pk = k;
    pstep = step;
    par ^= 1;
    __syncthreads();
    k += step;
  }
  store_l();
  __syncthreads();
  return nc;
}
