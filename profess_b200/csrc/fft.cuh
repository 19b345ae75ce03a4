// FP64 stages of the batched in-place FFT of dft.cuh.  The twiddles of stage s
// are a table W_{L_s}^{j0 r} in the order the butterflies read them (entry j0
// R_s + r), computed on the host in long double: a butterfly's R_s - 1 factors
// sit at fixed offsets from one address.
#pragma once
#include "dft.cuh"

namespace ofdft {

// v[r] *= w[r] (DIR < 0) or conj(w[r]) (DIR > 0), r = 1 .. R-1: a butterfly's
// stage twiddles.
template <typename T, int R, int DIR>
HD void twiddle_mul(cx<T>* v, const cx<T>* __restrict__ w) {
#pragma unroll
  for (int r = 1; r < R; ++r) v[r] = cmul(v[r], DIR < 0 ? w[r] : conj(w[r]));
}

// One in-place stage of radix R over ncols columns (mcols = magic32(ncols)):
// DIR = -1 forward (DFT, then twiddles), +1 inverse (conjugate twiddles,
// then inverse DFT).  w: the stage's twiddles.
template <typename T, int R, int DIR>
HD void ip_stage_r(cx<T>* __restrict__ buf, int ncols, unsigned mcols, int cs, int es, int n, int L, unsigned mm,
                   const cx<T>* __restrict__ wtab, int tid, int nthr) {
  const int m = L / R;
  const int total = (n / R) * ncols;
  const int ms = m * es;
  for (int w = tid; w < total; w += nthr) {
    const int bf = magic_div32(w, mcols), c = w - bf * ncols;
    const int blk = magic_div32(bf, mm), j0 = bf - blk * m;
    cx<T>* p = buf + c * cs + (blk * L + j0) * es;
    cx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[r * ms];
    if (DIR > 0 && m > 1) twiddle_mul<T, R, DIR>(v, wtab + j0 * R);
    Dft<T, R, DIR>::run(v);
    if (DIR < 0 && m > 1) twiddle_mul<T, R, DIR>(v, wtab + j0 * R);
#pragma unroll
    for (int r = 0; r < R; ++r) p[r * ms] = v[r];
  }
}

template <typename T, int DIR>
HD void ip_stage(cx<T>* buf, int ncols, unsigned mcols, int cs, int es, const StagePlan& p, int s, const cx<T>* tw,
                 int tid, int nthr) {
  const int n = p.n, L = p.L[s];
  const unsigned mm = p.m_magic[s];
  const cx<T>* w = tw + p.stw[s];
#define OFDFT_RADIX_DO(r) ip_stage_r<T, r, DIR>(buf, ncols, mcols, cs, es, n, L, mm, w, tid, nthr)
  OFDFT_RADIX_SWITCH(p.R[s])
#undef OFDFT_RADIX_DO
}

// One stage whose inputs come from src.ld(c, i) and whose outputs go to
// dst.st(c, i, v) (column c, position i), with the butterfly work split of
// ip_stage_r: a first forward stage can load straight from global memory, a
// last inverse stage store straight to it.
template <typename T, int R, int DIR, class Src, class Dst>
HD void ip_stage_io(const Src& src, const Dst& dst, int ncols, unsigned mcols, int n, int L, unsigned mm,
                    const cx<T>* __restrict__ wtab, int tid, int nthr) {
  const int m = L / R;
  const int total = (n / R) * ncols;
  for (int w = tid; w < total; w += nthr) {
    const int bf = magic_div32(w, mcols), c = w - bf * ncols;
    const int blk = magic_div32(bf, mm), j0 = bf - blk * m;
    const int base = blk * L + j0;
    cx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src.ld(c, base + r * m);
    if (DIR > 0 && m > 1) twiddle_mul<T, R, DIR>(v, wtab + j0 * R);
    Dft<T, R, DIR>::run(v);
    if (DIR < 0 && m > 1) twiddle_mul<T, R, DIR>(v, wtab + j0 * R);
#pragma unroll
    for (int r = 0; r < R; ++r) dst.st(c, base + r * m, v[r]);
  }
}

// Stage s of plan p through accessors (a switch over the radix).
template <typename T, int DIR, class Src, class Dst>
HD void ip_stage_acc(const Src& src, const Dst& dst, int ncols, unsigned mcols, const StagePlan& p, int s,
                     const cx<T>* tw, int tid, int nthr) {
  const int n = p.n, L = p.L[s];
  const unsigned mm = p.m_magic[s];
  const cx<T>* w = tw + p.stw[s];
#define OFDFT_RADIX_DO(r) ip_stage_io<T, r, DIR>(src, dst, ncols, mcols, n, L, mm, w, tid, nthr)
  OFDFT_RADIX_SWITCH(p.R[s])
#undef OFDFT_RADIX_DO
}

template <typename T, class Op>
HD void ip_stage_op(cx<T>* buf, int ncols, unsigned mcols, int cs, int es, const StagePlan& p, const Op& op, int tid,
                    int nthr) {
  const int n = p.n;
#define OFDFT_RADIX_DO(r) ip_stage_op_r<T, r>(buf, ncols, mcols, cs, es, n, op, tid, nthr)
  OFDFT_RADIX_SWITCH(p.R[p.nst - 1])
#undef OFDFT_RADIX_DO
}

// Full in-place transform of ncols columns (element i of column c at
// buf[c*cs + i*es]).  DIR = -1: forward, natural -> digit-reversed; DIR = +1:
// inverse, digit-reversed -> natural.  Every thread of the block must call
// it; the data must be complete in shared memory on entry (the caller's
// barrier), and the block synchronises after every stage, so the result is
// complete on return.
template <typename T, int DIR>
HD void fft_inplace(cx<T>* buf, int ncols, int cs, int es, const StagePlan& p, const cx<T>* tw, int tid, int nthr) {
  const unsigned mcols = magic32(ncols);
  if (DIR < 0) {
    for (int s = 0; s < p.nst; ++s) {
      ip_stage<T, -1>(buf, ncols, mcols, cs, es, p, s, tw, tid, nthr);
      BLOCK_SYNC();
    }
  } else {
    for (int s = p.nst - 1; s >= 0; --s) {
      ip_stage<T, 1>(buf, ncols, mcols, cs, es, p, s, tw, tid, nthr);
      BLOCK_SYNC();
    }
  }
}

// ------------------------------------------------------------ host planning
// Radix sequence of n (7-smooth, n <= 512): the fewest stages with radices
// up to rmax, then the smallest largest radix; largest radix first.  No heap
// use (the allocation-free entry point plans with it too).  Returns the
// number of stages, 0 if n has no such factorisation.  One table holds the
// sequences of every length (a search for each of an engine's 800 plans was a
// third of its creation).
constexpr int FFT_MAX_N = 512;
struct RadixTable {
  short first[FFT_MAX_RADIX + 1][FFT_MAX_N + 1];  // largest radix of the sequence of m with radices up to rmax (0: none)
  RadixTable() {
    static const int kR[] = {16, 15, 14, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    memset(first, 0, sizeof(first));
    for (int rmax = 2; rmax <= FFT_MAX_RADIX; ++rmax) {
      int st[FFT_MAX_N + 1], big[FFT_MAX_N + 1];
      for (int m = 0; m <= FFT_MAX_N; ++m) st[m] = big[m] = 1 << 20;
      st[1] = 0;
      big[1] = 0;
      for (int m = 2; m <= FFT_MAX_N; ++m)
        for (int R : kR) {
          if (R > rmax || m % R || st[m / R] >= (1 << 20)) continue;
          const int cs = st[m / R] + 1, cb = R > big[m / R] ? R : big[m / R];
          if (cs < st[m] || (cs == st[m] && cb < big[m])) { st[m] = cs; big[m] = cb; first[rmax][m] = (short)R; }
        }
    }
  }
};
inline int fft_radices(int n, int rmax, int* out) {
  static const RadixTable table;
  int k = 0;
  for (int m = n; m > 1; m /= table.first[rmax][m]) {
    if (!table.first[rmax][m]) return 0;
    out[k++] = table.first[rmax][m];
  }
  for (int a = 0; a < k; ++a)  // largest first
    for (int b = a + 1; b < k; ++b)
      if (out[b] > out[a]) { const int t = out[a]; out[a] = out[b]; out[b] = t; }
  return k;
}

// Entries of the stage twiddle tables of a plan, and the tables themselves:
// put(off, j) is called for every entry, whose value is exp(-2 pi i j / n).
// Fills p.stw from off0 on (even offsets); a stage of stride 1 has no table.
// Returns the end offset.
template <class Put>
inline int fft_stage_twiddles(StagePlan& p, int off0, Put put) {
  int off = off0;
  for (int s = 0; s < p.nst; ++s) {
    const int m = p.L[s] / p.R[s];
    p.stw[s] = off;
    if (m == 1) continue;
    for (int j0 = 0; j0 < m; ++j0)
      for (int r = 0; r < p.R[s]; ++r) put(off + j0 * p.R[s] + r, (int)((long long)j0 * r % p.L[s] * (p.n / p.L[s])));
    off += p.L[s] + (p.L[s] & 1);
  }
  return off;
}

// The x-inverse plan of a length: the pass runs at least two stages, so a
// one-stage plan gets a second stage of radix 1.
inline StagePlan x_plan(StagePlan p) {
  if (p.nst != 1) return p;
  p.nst = 2;
  p.R[1] = 1;
  p.L[1] = 1;
  p.m_magic[1] = magic32(1);
  p.stw[1] = p.stw[0];
  return p;
}

// Radix sequence of the x-forward pass: the pass keeps two blocks of its last
// stage in registers (x_last_split), so that stage's radix is 4 at most - or 1,
// a stage that only splits the rows - whatever the others are.  At 80
// registers a thread a radix of 5 or 6 spills 0.1 KB, 8 0.3 KB, 12 1.2 KB (16 x
// 96^3 FP64: 258 us with 6 4 4, 289 with 12 8; 8 x 64^3: 53 us with 4 4 4, 61 with
// 8 8; 2 x 105^3, 7 5 3: 59 us, 63 with last radices up to 8).
constexpr int XLAST_MAX = 4;
inline int xfwd_radices(int n, int rmax, int* out) {
  int rad[FFT_MAX_STAGES];
  int k = fft_radices(n, rmax, rad), big = rad[0];
  for (int s = 0; s < k; ++s) out[s] = rad[s];
  if (k == 1 || rad[k - 1] > XLAST_MAX) out[k++] = 1;
  for (int r = XLAST_MAX; r >= 2; --r) {
    if (n % r || n == r) continue;
    const int q = fft_radices(n / r, rmax, rad) + 1;
    if (q > k || (q == k && rad[0] >= big)) continue;
    for (int s = 0; s < q - 1; ++s) out[s] = rad[s];
    out[q - 1] = r;
    k = q;
    big = rad[0];
  }
  return k;
}

// Fill plan p of length n from its radix sequence (stage block lengths and
// magic numbers; the table offsets are the caller's), and the digit-reversal
// tables: perm[q] = frequency at position q after the forward transform,
// iperm[k] = position of frequency k.  No heap use.
inline void fft_plan_fill(FftPlan& p, int n, const int* radix, int nst, int* perm, int* iperm) {
  p.n = n;
  p.nst = nst;
  int L = n;
  for (int s = 0; s < nst; ++s) {
    p.R[s] = radix[s];
    p.L[s] = L;
    p.m_magic[s] = magic32(L / radix[s]);
    L /= radix[s];
  }
  for (int q = 0; q < n; ++q) {
    int k = 0, mult = 1, rem = q, len = n;
    for (int s = 0; s < nst; ++s) {
      const int m = len / radix[s];
      const int r = rem / m;
      k += mult * r;
      mult *= radix[s];
      rem -= r * m;
      len = m;
    }
    perm[q] = k;
    iperm[k] = q;
  }
}

}  // namespace ofdft
