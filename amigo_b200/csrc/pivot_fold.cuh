// Folds of the pivot search: the first largest |entry| of a column over the
// candidate rows and the largest over the others.  Included by ldl_factor.cu
// inside its namespace.

// What a warp keeps, and a CTA sends to the others, in a reduction: the bits
// of the largest |candidate entry| (h, l) and its position i (kNoPos: none),
// those of the largest |other entry| (th, tl), and a value of the row the
// step is about (wh, wl).  Non-negative doubles order like their bits, so the
// folds are integer maxima (redux.sync).
struct alignas(16) RowEntry {
  unsigned h, l, i, th, tl, wh, wl, pad;
};
constexpr unsigned kNoPos = 0x7fffffffu;

// First-argmax (h, l, i) and maximum (th, tl) of a warp, in every lane.
__device__ __forceinline__ void row_fold_max(unsigned& th, unsigned& tl) {
  const unsigned m = __reduce_max_sync(0xffffffffu, th);
  tl = __reduce_max_sync(0xffffffffu, th == m ? tl : 0u);
  th = m;
}
__device__ __forceinline__ void row_fold(RowEntry& e) {
  const unsigned FULL = 0xffffffffu;
  const unsigned mh = __reduce_max_sync(FULL, e.h);
  const unsigned ml = __reduce_max_sync(FULL, e.h == mh ? e.l : 0u);
  e.i = __reduce_min_sync(FULL, e.h == mh && e.l == ml ? e.i : kNoPos);
  e.h = mh;
  e.l = ml;
  row_fold_max(e.th, e.tl);
}
__device__ __forceinline__ double row_bits(unsigned h, unsigned l) {
  return __hiloint2double((int)h, (int)l);
}
// |a| at position p into the argmax (cand) or into the maximum (other); a NaN
// counts as no entry.  (Selects, not branches.)
__device__ __forceinline__ void row_argmax(RowEntry& e, double a, int p, bool cand) {
  const unsigned h = (unsigned)__double2hiint(a), l = (unsigned)__double2loint(a);
  const unsigned long long x = ((unsigned long long)h << 32) | l;
  const unsigned long long y = ((unsigned long long)e.h << 32) | e.l;
  const bool gt = cand && a == a && (x > y || (x == y && (unsigned)p < e.i));
  e.h = gt ? h : e.h;
  e.l = gt ? l : e.l;
  e.i = gt ? (unsigned)p : e.i;
}
__device__ __forceinline__ void row_max(RowEntry& e, double a, bool other) {
  const unsigned h = (unsigned)__double2hiint(a), l = (unsigned)__double2loint(a);
  const unsigned long long x = ((unsigned long long)h << 32) | l;
  const unsigned long long y = ((unsigned long long)e.th << 32) | e.tl;
  const bool gt = other && a == a && x > y;
  e.th = gt ? h : e.th;
  e.tl = gt ? l : e.tl;
}

