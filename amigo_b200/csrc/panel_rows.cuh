// Large-front panel with one row of the front per thread, the panel's L
// entries of the row in registers.  Included by ldl_factor.cu inside its
// namespace (the pivot rule, the warp folds and the HBM-panel form are
// there).
//
// A panel is a chain of dependent pivot steps, so a step's latency is what
// counts, not its bandwidth.  Measured on 1,100-row fronts (cycles of a step
// without an interchange / with a second column and an interchange / a delayed
// pivot): the shared-memory cluster panel (k_big_panel_cl) 5,000 / 12,000 /
// 45,000, this one 2,300 / 5,300 / 5,300.  What changed:
//   * a thread keeps L[r, 0:32] of its row in registers, so that a column
//     build is an unrolled run of multiply-adds over the W row of the
//     column, read from shared memory (one broadcast for all lanes);
//   * interchanges and delays move nothing: every row stays with its thread
//     and in its place in F, and only the position a row stands for changes
//     (pos, and for the candidates the arrays `sl` and `ph`).  The entries of
//     the trailing block that end up elsewhere are moved together when
//     kRowMoves positions have changed and at the end of the panel, the rows
//     left of the panel and the variable list at its end;
//   * what the CTAs tell each other goes by stores that report to an mbarrier
//     (st.async) instead of cluster barriers: a reduction is one message per
//     pair of CTAs, and the next candidate's W row comes with it;
//   * the candidate columns are loaded three steps ahead.
// The rows are dealt to the CTAs of a cluster of CS in groups of 32, as in
// k_big_panel_cl, and every entry gets the same operations in the same order
// as there: the results are the same bit for bit.  One factorization, before
// (one-CTA panels to 768 rows, k_big_panel_cl above) and after: 2D SIMP 32x16
// 4.57 -> 2.97 ms, 61x27 10.26 -> 5.94, 128x64 25.6 -> 16.9, 3D 20x10x10
// 82.5 -> 46.8.  A step is bound by the latency of ~490 instructions of one
// warp, the panel's end included (ncu, 1,120 rows on 8 CTAs: 8.8 cycles from one
// to the next, no pipe above 20%).
constexpr int kRowThreads = 256;

constexpr int kRowMoves = 16;  // positions moved per flush

// Messages of a step: the reduction over the candidate column together with
// the next candidate's W row (RED), the W row of column imax (IMAX), the
// reduction over it (RED2), and the next candidate's W row when it was not
// the row sent ahead (NEXT).  Each has its buffer and mbarrier per step
// parity: it is written again two steps later, after a reduction every CTA
// took part in, so no CTA still reads it.
enum : int { ROW_RED = 0, ROW_IMAX = 1, ROW_RED2 = 2, ROW_NEXT = 3 };

template <class T, int PT, int CS>
struct RowCtl {
  static constexpr int NW = PT / 32;
  unsigned long long bar[2][4];   // mbarriers by parity and message
  RowEntry ent[2][2][CS];         // parity; RED, RED2
  alignas(16) T y[2][NB];         // the candidate's W row by step parity
  alignas(16) T yi[NB];           // column imax's W row
  // the warps' parts of the CTA's entries, by parity and reduction, and the
  // values of row k (its diagonal) and of row imax (diagonal, entry k)
  RowEntry we[2][2][NW];
  double ww[2][3];
  msg::Leave leave;
  int kind[NB];
  int nm, nr;
  int mp[kRowMoves], mq[kRowMoves];             // moved positions and where their entries are
};

template <int CS>
__device__ __forceinline__ void row_barrier() {
  if constexpr (CS == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;\n"
                 "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
}

// A value that is the same in every lane of a warp, in a form that the compiler
// knows to be so (a warp reduction): branches on it need no reconvergence, and
// what is computed from it stays in uniform registers.
__device__ __forceinline__ int row_uniform(int v) {
  return __reduce_max_sync(0xffffffffu, v);
}

// The panel's L entries of a thread's rows: complete groups of eight columns
// in g, the last columns in t (column j at t[j % 8], zero past the panel's
// columns).  An entry is set by selects over t alone; a store at a variable
// index would put the array in local memory.
template <class T, int RPT>
struct RowL {
  T g[RPT][NB - 8], t[RPT][8];
};

// 8 entries of y (16-byte aligned) against the columns' L entries l.
template <class T>
__device__ __forceinline__ void row_load8(T (&v)[8], const T* y) {
  constexpr int Q = 8 * sizeof(T) / 16;
  int4 raw[Q];
#pragma unroll
  for (int u = 0; u < Q; u++) raw[u] = reinterpret_cast<const int4*>(y)[u];
  memcpy(v, raw, sizeof(v));
}

// acc[i] -= sum_{j < kw} L[i][j] y[j] in the order of sw_apply_panel (column
// j into partial j mod 4); y[j] = 0 for kw <= j.
template <class T, int RPT>
__device__ __forceinline__ void row_apply(const T* y, int kw, const RowL<T, RPT>& L,
                                          T (&acc)[RPT]) {
  T s[RPT][4];
#pragma unroll
  for (int i = 0; i < RPT; i++)
#pragma unroll
    for (int q = 0; q < 4; q++) s[i][q] = T(0);
  T v[8];
#pragma unroll
  for (int g = 0; g + 8 < NB; g += 8) {
    if (g + 8 <= kw) {
      row_load8<T>(v, y + g);
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int i = 0; i < RPT; i++) s[i][u & 3] = fma(L.g[i][g + u], v[u], s[i][u & 3]);
    }
  }
  if (kw & 7) {
    row_load8<T>(v, y + (kw & ~7));
#pragma unroll
    for (int u = 0; u < 8; u++)
#pragma unroll
      for (int i = 0; i < RPT; i++) s[i][u & 3] = fma(L.t[i][u], v[u], s[i][u & 3]);
  }
  sum4_apply<T, RPT>(acc, s);
}

// L entries of column kw.
template <class T, int RPT>
__device__ __forceinline__ void row_set(RowL<T, RPT>& L, int kw, const T (&v)[RPT]) {
#pragma unroll
  for (int u = 0; u < 8; u++)
#pragma unroll
    for (int i = 0; i < RPT; i++) L.t[i][u] = u == (kw & 7) ? v[i] : L.t[i][u];
  if ((kw & 7) == 7 && kw < NB - 1) {
#pragma unroll
    for (int g = 0; g + 8 < NB; g += 8) {
      // (opaque to the compiler: it would merge the groups into a store at
      // a variable index)
      int h;
      asm volatile("and.b32 %0, %1, -8;" : "=r"(h) : "r"(kw));
      if (h == g) {
#pragma unroll
        for (int u = 0; u < 8; u++)
#pragma unroll
          for (int i = 0; i < RPT; i++) L.g[i][g + u] = L.t[i][u];
      }
    }
#pragma unroll
    for (int u = 0; u < 8; u++)
#pragma unroll
      for (int i = 0; i < RPT; i++) L.t[i][u] = T(0);
  }
}

// Shared memory of the kernel: W of the CTA's rows (NB columns of leading
// dimension lld, odd, so that a row's columns fall on distinct banks), the
// candidates' rows and places, and the list of moved positions.
template <class T>
__host__ __device__ __forceinline__ size_t row_smem(int lld, int ncap) {
  return (size_t)NB * lld * sizeof(T) + 3 * (size_t)ncap * sizeof(unsigned short);
}

template <class T, int PT, int RPT, int CS>
__device__ void panel_factor_rows(T* F, int ld, T* Wg, int n, bool root, int* vars,
                                  int* fsperm, double ustab, double pivot_tol,
                                  int* status, int polls,
                                  RowCtl<T, PT, CS>& c, T* Ws, int lld,
                                  unsigned short* sl, unsigned short* ph,
                                  unsigned short* lst, int cr, int& k_, int& nc_,
                                  int& kw_) {
  constexpr int NW = PT / 32, MV = kRowMoves;
  constexpr unsigned kYBytes = NB * sizeof(T), kRedBytes = CS * sizeof(RowEntry);
  const unsigned FULL = 0xffffffffu;
  // (read once: the compiler would read the special registers again in every
  // step)
  int tid;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
  const int lane = tid & 31, warp = row_uniform(tid >> 5);
  const bool lead = cr == 0 && tid == 0;
  int k = row_uniform(k_), nc = row_uniform(nc_), kw = 0;
  const int kstart = k, nc0 = nc, cld = n - kstart;
  // A row: its local index, the position it stands for (-1: none; a row is
  // live while pos >= k) and its place in F.  Candidate position p: its row
  // sl[p - kstart] and place ph[p - kstart], relative to kstart.
  int lr[RPT], pos[RPT], phys[RPT];
  RowL<T, RPT> L;
#pragma unroll
  for (int i = 0; i < RPT; i++) {
    lr[i] = 32 * (warp + NW * i) + lane;
    const int rel = 32 * (CS * (warp + NW * i) + cr) + lane;
    pos[i] = phys[i] = rel < cld ? kstart + rel : -1;
#pragma unroll
    for (int j = 0; j < NB - 8; j++) L.g[i][j] = T(0);
#pragma unroll
    for (int j = 0; j < 8; j++) L.t[i][j] = T(0);
  }
  for (int p = tid; p < nc0 - kstart; p += PT) sl[p] = ph[p] = (unsigned short)p;
  for (int t = tid; t < 2 * NB; t += PT) c.y[t / NB][t % NB] = T(0);
  // The W column in shared memory of the panel's column j: pc of lane j for
  // the pivots taken, pa and pb for the candidate column and column imax (an
  // imax 1x1 pivot takes the column built second).
  int pc = lane, pa = 0, pb = 1;
  unsigned phase = 0;
  if constexpr (CS > 1) {
    if (tid < 8) msg::init(&c.bar[tid >> 2][tid & 3]);
    msg::leave_init(c.leave);
    msg::init_done();
  }
  // every CTA of the cluster has started and its mbarriers are set up before
  // anything is sent to it
  row_barrier<CS>();
  // a message has arrived (CS 1: the stores of the CTA's warps are published)
  auto wait = [&](int par, int m) {
    if constexpr (CS == 1) __syncthreads();
    else {
      // (phase: the bits of the mbarriers' phases, one per mbarrier)
      const int bit = 4 * par + m;
      msg::wait(&c.bar[par][m], (phase >> bit) & 1u, polls, c.leave, status, ST_WAIT);
      phase ^= 1u << bit;
    }
  };
  auto expect = [&](int par, int m, unsigned bytes) {
    if (CS > 1 && tid == 0) msg::expect(&c.bar[par][m], bytes);
  };
  auto load_pos = [&](int p, T (&dst)[RPT]) {
    const int q = kstart + ph[p - kstart];
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const int hi = max(phys[i], q), lo = min(phys[i], q);
      dst[i] = pos[i] >= k ? __ldcg(F + hi + (size_t)lo * ld) : T(0);
    }
  };
  // the W row (ncol entries, then zeros) of row q into every CTA's `dst`, by
  // the row's warp
  auto send_row = [&](int q, int ncol, T* dst, int par, int m) {
    const int r = cl_lrow<CS>(q);
    if (cl_owner<CS>(q) != cr || ((r >> 5) % NW) != warp) return;
    const T v = lane < ncol ? Ws[(size_t)pc * lld + r] : T(0);
    if constexpr (CS == 1) {
      dst[lane] = v;
    } else {
#pragma unroll
      for (int t = 0; t < CS; t++)
        msg::send(msg::remote(dst + lane, t), msg::remote(&c.bar[par][m], t), v);
    }
  };
  // this CTA's entry of a reduction to every CTA (set 0: the candidate column,
  // 1: column imax, a maximum and two values of row imax): the warps' folds,
  // a barrier, warp 0 folds them
  auto send_red = [&](int par, int set, RowEntry e) {
    if (set == 0) row_fold(e);
    else row_fold_max(e.th, e.tl);
    if (lane == 0) {
      if (set == 0) reinterpret_cast<uint4*>(&c.we[par][0][warp])[0] = make_uint4(e.h, e.l, e.i, e.th);
      else c.we[par][1][warp].th = e.th;
      c.we[par][set][warp].tl = e.tl;
    }
    __syncthreads();
    if (CS > 1 && warp == 0) {
      const RowEntry& w = c.we[par][set][lane < NW ? lane : 0];
      if (set == 0) {
        const uint4 x = reinterpret_cast<const uint4*>(&w)[0];
        e.h = x.x;
        e.l = x.y;
        e.i = x.z;
        e.th = x.w;
      } else {
        e.th = w.th;
      }
      e.tl = w.tl;
      const double v = c.ww[par][set], v2 = c.ww[par][2];
      if (set == 0) {
        row_fold(e);
      } else {
        row_fold_max(e.th, e.tl);
        e.h = (unsigned)__double2hiint(v2);
        e.l = (unsigned)__double2loint(v2);
      }
      if (lane < CS) {
        const unsigned dst = msg::remote(&c.ent[par][set][cr], lane);
        const unsigned bar = msg::remote(&c.bar[par][set ? ROW_RED2 : ROW_RED], lane);
        msg::send(dst, bar, make_uint4(e.h, e.l, e.i, e.th));
        msg::send(dst + 16, bar, make_uint4(e.tl, (unsigned)__double2hiint(v),
                                            (unsigned)__double2loint(v), 0u));
      }
    }
  };
  // the CTAs' entries (CS 1: the warps'), a lane each
  auto take_red = [&](int par, int set) -> RowEntry {
    constexpr int N = CS == 1 ? NW : CS;
    const RowEntry* e = CS == 1 ? c.we[par][set] : c.ent[par][set];
    return e[lane < N ? lane : 0];
  };
  // the rows' entries of a column to W column q
  auto store_w = [&](int q, const T (&v)[RPT]) {
    T* w = Ws + (size_t)q * lld;
#pragma unroll
    for (int i = 0; i < RPT; i++)
      if (pos[i] >= k) w[lr[i]] = v[i];
    __syncwarp();
  };
  auto swap_pos = [&](int a, int b) {
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      if (pos[i] == a) pos[i] = b;
      else if (pos[i] == b) pos[i] = a;
    }
    // (every read of the two entries in this step is done: the reduction over
    // column imax had a barrier after them)
    if (tid == 0) {
      const unsigned short s = sl[a - kstart], q = ph[a - kstart];
      sl[a - kstart] = sl[b - kstart];
      ph[a - kstart] = ph[b - kstart];
      sl[b - kstart] = s;
      ph[b - kstart] = q;
    }
    __syncthreads();
  };
  // Move the entries of the live block whose positions changed to their
  // place: all loads of the cluster, a barrier, all stores.  (The sources are
  // in columns >= kstart that no store of the panel has touched yet.)
  int moves = 0;  // bound on the live candidate positions that changed
  auto flush = [&]() {
    if (tid == 0) c.nm = 0;
    __syncthreads();
    for (int p = k + tid; p < nc0; p += PT)
      if (kstart + ph[p - kstart] != p) {
        const int t = atomicAdd(&c.nm, 1);
        c.mp[t] = p;
        c.mq[t] = kstart + ph[p - kstart];
      }
    __syncthreads();
    const int nm = c.nm;
    // (loops over groups of eight, the values in local memory: this runs once
    // or twice in a panel, and unrolled code would push the step's own out of
    // the instruction cache)
    T v[RPT * MV];
#pragma unroll 1
    for (int m0 = 0; m0 < nm; m0 += 8) {
      T x[8][RPT];
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          const int q = m0 + u < nm ? c.mq[m0 + u] : -1;
          const int hi = max(phys[i], q), lo = min(phys[i], q);
          x[u][i] = q >= 0 && pos[i] >= k ? __ldcg(F + hi + (size_t)lo * ld) : T(0);
        }
#pragma unroll
      for (int u = 0; u < 8; u++)
#pragma unroll
        for (int i = 0; i < RPT; i++) v[(m0 + u) * RPT + i] = x[u][i];
    }
    row_barrier<CS>();
#pragma unroll 1
    for (int m = 0; m < nm; m++)
#pragma unroll
      for (int i = 0; i < RPT; i++)
        if (pos[i] >= k) {
          const int p = c.mp[m], q = pos[i];
          // an entry between two moved positions: from the later one's row
          if (q >= p || phys[i] == q)
            F[max(p, q) + (size_t)min(p, q) * ld] = v[m * RPT + i];
        }
#pragma unroll
    for (int i = 0; i < RPT; i++)
      if (pos[i] >= k) phys[i] = pos[i];
    if (tid < nm) ph[c.mp[tid] - kstart] = (unsigned short)(c.mp[tid] - kstart);
    row_barrier<CS>();
    moves = 0;
  };
  // the candidate columns at positions k .. k + 2 (rows s0 .. s2); at the
  // start of a step the one at k + 3 is started too
  T cur[RPT], n1[RPT], n2[RPT], n3[RPT];
  int s0 = -1, s1 = -1, s2 = -1, s3 = -1;
  auto copy = [&](T (&d)[RPT], const T (&x)[RPT]) {
#pragma unroll
    for (int i = 0; i < RPT; i++) d[i] = x[i];
  };
  // after a step with an interchange or two columns: the columns held are
  // kept, the others loaded
  auto refill = [&]() {
    T o0[RPT], o1[RPT], o2[RPT], o3[RPT];
    copy(o0, cur);
    copy(o1, n1);
    copy(o2, n2);
    copy(o3, n3);
    const int t0 = s0, t1 = s1, t2 = s2, t3 = s3;
    // (the three loads are in flight together)
    auto pick = [&](int p, int& s, T (&dst)[RPT]) {
      s = p < nc ? row_uniform(sl[p - kstart]) : -1;
      if (s < 0) return;
      if (s == t0) copy(dst, o0);
      else if (s == t1) copy(dst, o1);
      else if (s == t2) copy(dst, o2);
      else if (s == t3) copy(dst, o3);
      else load_pos(p, dst);
    };
    pick(k, s0, cur);
    pick(k + 1, s1, n1);
    pick(k + 2, s2, n2);
  };
#pragma unroll
  for (int i = 0; i < RPT; i++) cur[i] = n1[i] = n2[i] = n3[i] = T(0);
  refill();
  int par = 0;
  // the columns held are those of the positions from k on, and the candidate's
  // W row is in c.y[par] (kw 0: zeros) or on its way with the last reduction
  bool ahead = true;
  for (;;) {
    const bool more = kw < NB - 1 && k < nc;
    if (!more || !ahead) {
      if (more) send_row(row_uniform(sl[k - kstart]), kw, c.y[par], par, ROW_NEXT);
      if (moves > (more ? MV - 2 : 0)) flush();
      if (!more) break;
      expect(par, ROW_NEXT, kYBytes);
      refill();
      wait(par, ROW_NEXT);
    }
    expect(par, ROW_RED, kRedBytes + (s1 >= 0 ? kYBytes : 0u));
    s3 = k + 3 < nc ? row_uniform(sl[k + 3 - kstart]) : -1;
    if (s3 >= 0) load_pos(k + 3, n3);
    T acc[RPT];
    copy(acc, cur);
    row_apply<T, RPT>(c.y[par], kw, L, acc);
    store_w(pa, acc);
    if (lane == kw) pc = pa;
    // the next candidate's W row, in case this step takes a 1x1 pivot
    // without an interchange, and the candidate column's reduction
    if (CS == 1 && s1 >= 0) send_row(s1, kw + 1, c.y[par ^ 1], par, ROW_RED);
    RowEntry e{0u, 0u, kNoPos, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const double a = fabs((double)acc[i]);
      if (pos[i] == k) c.ww[par][0] = (double)acc[i];
      row_argmax(e, a, pos[i], pos[i] > k && pos[i] < nc);
      row_max(e, a, pos[i] >= nc);
    }
    send_red(par, 0, e);
    // (after the CTA's entry: warp 0 folds while the row's warp sends it)
    if (CS > 1 && s1 >= 0) send_row(s1, kw + 1, c.y[par ^ 1], par, ROW_RED);
    if constexpr (CS > 1) wait(par, ROW_RED);
    e = take_red(par, 0);
    const double wkk = CS == 1 ? c.ww[par][0]
                               : row_bits(c.ent[par][0][cl_owner<CS>(s0)].wh,
                                          c.ent[par][0][cl_owner<CS>(s0)].wl);
    const T dinv = T(1) / T(wkk);  // the 1x1 pivot's, ahead of the decision
    row_fold(e);
    const double abswik = row_bits(e.h, e.l), ctail = row_bits(e.th, e.tl);
    const bool tails = e.th > e.h || (e.th == e.h && e.tl > e.l);
    const double colmax = tails ? ctail : abswik;
    int imax = (int)e.i;
    if (imax >= nc || imax <= k) {
      if (k + 1 < nc && lead) atomicOr(status, ST_NAN);
      imax = (k + 1 < n) ? k + 1 : k;
    }
    // the decision as a word: step, zero pivot, imax 1x1, pivot at imax
    int code = plain_pivot(root, wkk, colmax, ustab, pivot_tol) ? 1 : 0;
    code = row_uniform(code);
    T a2[RPT];
    ImaxColumn ic{0.0, 0.0, 0.0};
    if (!code) {
      if (row_uniform(needs_imax(root, k, nc, wkk, abswik, ctail, ustab, pivot_tol))) {
        // column imax as the panel's column kw + 1; its owner sends its
        // diagonal and the candidate column's entry in row imax
        const int q = row_uniform(sl[imax - kstart]);
        send_row(q, kw, c.yi, par, ROW_IMAX);
        expect(par, ROW_IMAX, kYBytes);
        expect(par, ROW_RED2, kRedBytes);
        load_pos(imax, a2);
        wait(par, ROW_IMAX);
        row_apply<T, RPT>(c.yi, kw, L, a2);
        store_w(pb, a2);
        RowEntry f{0u, 0u, kNoPos, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          const double a = fabs((double)a2[i]);
          if (pos[i] == imax) {
            c.ww[par][1] = (double)acc[i];
            c.ww[par][2] = (double)a2[i];
          }
          row_max(f, a, pos[i] >= k && pos[i] != imax);
        }
        send_red(par, 1, f);
        if constexpr (CS > 1) wait(par, ROW_RED2);
        f = take_red(par, 1);
        row_fold_max(f.th, f.tl);
        ic.rowmax = row_bits(f.th, f.tl);
        if constexpr (CS == 1) {
          ic.wik = c.ww[par][1];
          ic.wii = c.ww[par][2];
        } else {
          const RowEntry& o = c.ent[par][1][cl_owner<CS>(q)];
          ic.wik = row_bits(o.wh, o.wl);
          ic.wii = row_bits(o.h, o.l);
        }
      }
      const PivotChoice pv = choose_pivot(root, k, nc, wkk, imax, abswik, ctail, ustab,
                                          pivot_tol, [&]() { return ic; });
      code = row_uniform(pv.step | (pv.zero ? 4 : 0) | (pv.imax_1x1 ? 8 : 0) |
                         (pv.step && pv.kpiv == imax ? 16 : 0));
    }
    const int step = code & 3;
    const bool imax_1x1 = (code & 8) != 0;
    if (step == 0) {
      // delay candidate k: it moves to the end of the candidate set
      if (k < nc - 1) {
        swap_pos(k, nc - 1);
        moves += 2;
      }
      nc -= 1;
      par ^= 1;
      ahead = false;
      continue;
    }
    const int kpiv = code & 16 ? imax : k;
    const bool swapped = kpiv != k + step - 1;
    if (swapped) {
      swap_pos(k + step - 1, kpiv);
      moves += 1;
    }
    // the pivot block and the L columns of the pivot, with the expressions of
    // the other panel kernels
    T l[RPT], l1[RPT];
    if (step == 1) {
      const T d = imax_1x1 ? T(ic.wii) : T(wkk);
      if (!isfinite((double)d) && lead) atomicOr(status, ST_NAN);
      const T ainv = code & 4 ? T(0) : (imax_1x1 ? T(1) / d : dinv);
      if (tid == 0) c.kind[kw] = 0;
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const T w = imax_1x1 ? a2[i] : acc[i];
        l[i] = sw_l(w, w, ainv, T(0));
      }
      if (imax_1x1) {
        // column imax is the pivot column
        if (lane == kw) pc = pb;
      } else {
        pa = pb;
      }
    } else {
      const Coef2 q = pivot2_coeffs<T>(T(wkk), T(ic.wik), T(ic.wii));
      if (!q.finite && lead) atomicOr(status, ST_NAN);
      if (tid == 0) {
        c.kind[kw] = 1;
        c.kind[kw + 1] = 2;
      }
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        l[i] = sw_l(acc[i], a2[i], T(q.i00), T(q.i10));
        l1[i] = sw_l(a2[i], acc[i], T(q.i11), T(q.i01));
      }
      if (lane == kw + 1) pc = pb;
      pa = kw + 2;
    }
    row_set<T, RPT>(L, kw, l);
    if (step == 2) row_set<T, RPT>(L, kw + 1, l1);
    k += step;
    kw += step;
    pb = kw + 1;
    par ^= 1;
    ahead = step == 1 && !swapped;
    if (ahead) {
      copy(cur, n1);
      copy(n1, n2);
      copy(n2, n3);
      s0 = s1;
      s1 = s2;
      s2 = s3;
    }
  }
  // --- entries of the trailing block to their place; then, once no CTA reads
  // the panel's columns of F any more, L and D to F and W below the panel to
  // HBM, each CTA for its own rows
  row_barrier<CS>();
  // (no CTA sends to another from here on)
  if constexpr (CS > 1)
    if (__any_sync(FULL, *(volatile int*)&c.leave.dead))
      msg::leave(&c.leave, status, ST_WAIT);
  // D and W from shared memory, then L through it (each thread its own rows),
  // eight columns' loads before their stores
  constexpr int WB8 = 8 / RPT;
#pragma unroll 1
  for (int j0 = 0; j0 < kw; j0 += WB8) {
    T w[WB8][RPT];
#pragma unroll
    for (int u = 0; u < WB8; u++) {
      const T* w0 = Ws + (size_t)__shfl_sync(FULL, pc, (j0 + u) & 31) * lld;
#pragma unroll
      for (int i = 0; i < RPT; i++) w[u][i] = pos[i] >= kstart ? w0[lr[i]] : T(0);
    }
#pragma unroll
    for (int u = 0; u < WB8; u++) {
      const int col = kstart + j0 + u;
      const bool first = c.kind[(j0 + u) & 31] == 1;  // of a 2x2 pivot
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const int p = pos[i];
        if (j0 + u < kw) {
          if (p >= k) Wg[p + (size_t)(j0 + u) * ld] = w[u][i];
          if (p == col || (first && p == col + 1)) F[p + (size_t)col * ld] = w[u][i];
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RPT; i++)
    if (pos[i] >= kstart) {
#pragma unroll
      for (int j = 0; j < NB - 8; j++) Ws[(size_t)j * lld + lr[i]] = L.g[i][j];
#pragma unroll
      for (int u = 0; u < 8; u++) Ws[(size_t)((NB - 8) + u) * lld + lr[i]] = L.t[i][u];
    }
#pragma unroll 1
  for (int j0 = 0; j0 < kw; j0 += WB8) {
    T w[WB8][RPT];
#pragma unroll
    for (int u = 0; u < WB8; u++) {
      const int j = j0 + u;
      const T* l0 = Ws + (size_t)(j < (kw & ~7) && j < NB - 8 ? j : NB - 8 + (j & 7)) * lld;
#pragma unroll
      for (int i = 0; i < RPT; i++) w[u][i] = pos[i] >= kstart ? l0[lr[i]] : T(0);
    }
#pragma unroll
    for (int u = 0; u < WB8; u++) {
      const int col = kstart + j0 + u, past = col + (c.kind[(j0 + u) & 31] == 1 ? 1 : 0);
#pragma unroll
      for (int i = 0; i < RPT; i++)
        if (j0 + u < kw && pos[i] > past) F[pos[i] + (size_t)col * ld] = w[u][i];
    }
  }
  // the panel's interchanges of the columns left of it, of the variable list
  // and of the fully-summed permutation: position p takes row sl[p - kstart]
  if (tid == 0) c.nr = 0;
  __syncthreads();
  for (int p = tid; p < nc0 - kstart; p += PT)
    if (sl[p] != p) lst[atomicAdd(&c.nr, 1)] = (unsigned short)p;
  __syncthreads();
  const int nr = c.nr;
  if (nr > 0) {
    if (cr == 0) {
      // (W is written out: its shared memory stages the entries)
      int* sv = reinterpret_cast<int*>(Ws);
      for (int t = tid; t < nr; t += PT) {
        sv[2 * t] = vars[kstart + sl[lst[t]]];
        sv[2 * t + 1] = fsperm[kstart + sl[lst[t]]];
      }
      __syncthreads();
      for (int t = tid; t < nr; t += PT) {
        vars[kstart + lst[t]] = sv[2 * t];
        fsperm[kstart + lst[t]] = sv[2 * t + 1];
      }
      __syncthreads();
    }
    if (nr <= 64) {
      const bool h0 = lane < nr, h1 = lane + 32 < nr;
      const int d0 = h0 ? kstart + lst[lane] : 0, d1 = h1 ? kstart + lst[lane + 32] : 0;
      const int q0 = h0 ? kstart + sl[d0 - kstart] : 0;
      const int q1 = h1 ? kstart + sl[d1 - kstart] : 0;
      constexpr int CB = 8;
      for (int j0 = (cr * NW + warp) * CB; j0 < kstart; j0 += CS * NW * CB) {
        T v0[CB], v1[CB];
#pragma unroll
        for (int u = 0; u < CB; u++) {
          const T* Fj = F + (size_t)(j0 + u) * ld;
          const bool in = j0 + u < kstart;
          v0[u] = in && h0 ? __ldcg(Fj + q0) : T(0);
          v1[u] = in && h1 ? __ldcg(Fj + q1) : T(0);
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < CB; u++) {
          if (j0 + u >= kstart) break;
          T* Fj = F + (size_t)(j0 + u) * ld;
          if (h0) Fj[d0] = v0[u];
          if (h1) Fj[d1] = v1[u];
        }
      }
    } else {
      // many delays in one panel: a column at a time through shared memory,
      // by as many warps as have room for one
      const int room = NB * lld;
      const int nw = min(NW, room / nr);
      T* st = Ws + (size_t)warp * nr;
      if (warp < nw)
        for (int j = cr * nw + warp; j < kstart; j += CS * nw) {
          T* Fj = F + (size_t)j * ld;
          for (int t = lane; t < nr; t += 32) st[t] = __ldcg(Fj + kstart + sl[lst[t]]);
          __syncwarp();
          for (int t = lane; t < nr; t += 32) Fj[kstart + lst[t]] = st[t];
          __syncwarp();
        }
    }
  }
  // the panel's pivot kinds (2x2 pivots' variables encoded -(v + 1))
  if (cr == 0 && tid < kw) {
    const int col = kstart + tid, kd = c.kind[tid];
    vars[3 * ld + col] = kd;
    if (kd != 0) vars[col] = -(vars[col] + 1);
  }
  k_ = k;
  nc_ = nc;
  kw_ = kw;
}

// One cluster of CS CTAs per front (CS 1: one CTA).  Fronts of more than
// fit_rows rows, or past the launch's rows, take the HBM-panel form on CTA 0.
template <class T, int PT, int RPT, int CS>
__global__ void __launch_bounds__(PT, 1)
k_big_panel_rows(DevicePlan d, const int* __restrict__ nodes, double ustab,
                 double pivot_tol, int lld, int ncap, int fit_rows) {
  pdl_enter();
  __shared__ RowCtl<T, PT, CS> c;
  __shared__ CtlT<PT> ctl;
  extern __shared__ double row_raw[];
  const bool skip = big_skip(d);
  int cr = 0;
  if constexpr (CS > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(cr));
  cr = row_uniform(cr);
  const int node = nodes[blockIdx.x / CS];
  int* st = d.pstate + 4 * node;
  int k = st[0], nc = st[1];
  // (pools run out in earlier launches only; a wait, also in another cluster of
  // this one, so that the CTAs of a cluster may read different answers: they
  // start all the same, and those that know give up at their first wait)
  const int over = __syncthreads_or(skip);
  if (over && (CS == 1 || pools_out(d))) return;
  if (k >= nc) {
    if (cr == 0 && threadIdx.x == 0) st[3] = 0;
    return;
  }
  const int f = d.f[node];
  const int fs = d.ns[node] + d.ndin[node];
  T* F = reinterpret_cast<T*>(d.fpool) + d.foff[node];
  T* W = F + (size_t)f * f;
  int* fvars = d.ipool + d.ioff[node];
  const int kstart = k, cld = f - kstart;
  int kw = 0;
  T* Ws = reinterpret_cast<T*>(row_raw);
  unsigned short* sl = reinterpret_cast<unsigned short*>(Ws + (size_t)NB * lld);
  if (cld <= fit_rows && cld <= CS * PT * RPT && cl_local_rows<CS>(cld) < lld &&
      nc - kstart <= ncap) {
    // (CTA 0 stores the state below only after the cluster's first barrier,
    // when every CTA has read it)
    panel_factor_rows<T, PT, RPT, CS>(F, f, W, f, fs == f, fvars, fvars + f, ustab,
                                      pivot_tol, d.status, over ? 0 : d.wait_polls, c, Ws, lld,
                                      sl, sl + ncap,
                                      sl + 2 * ncap, cr, k, nc, kw);
  } else {
    row_barrier<CS>();
    if (cr != 0) return;
    if (threadIdx.x == 0) atomicAdd(d.scratch_int + 5, 1);
    panel_factor<T, PT>(F, f, W, f, f, fs == f, fvars, fvars + f, ustab, pivot_tol,
                        d.status, ctl, k, nc, kw);
  }
  if (cr == 0 && threadIdx.x == 0) {
    st[0] = k;
    st[1] = nc;
    st[2] = kstart;
    st[3] = kw;
  }
}
