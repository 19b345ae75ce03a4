// FP32 stages of the batched in-place FFT of ../dft.cuh.  The twiddles are the
// n-th roots of unity exp(-2 pi i e / n), e < n, computed on the host in long
// double; W_{L_s}^{e} is root[e n / L_s].
#pragma once
#include "../dft.cuh"

namespace ofdft {
namespace f32 {

// One in-place stage of radix R over ncols columns (mcols = magic32(ncols)):
// DIR = -1 forward (DFT, then twiddles), +1 inverse (conjugate twiddles,
// then inverse DFT).  tstep = n / L.
template <typename T, int R, int DIR>
HD void ip_stage_r(cx<T>* __restrict__ buf, int ncols, unsigned mcols, int cs, int es, int n, int L, unsigned mm,
                   const cx<T>* __restrict__ roots, int tid, int nthr) {
  const int m = L / R;
  const int total = (n / R) * ncols;
  const int tstep = n / L;
  const int ms = m * es;
  for (int w = tid; w < total; w += nthr) {
    const int bf = magic_div32(w, mcols), c = w - bf * ncols;
    const int blk = magic_div32(bf, mm), j0 = bf - blk * m;
    cx<T>* p = buf + c * cs + (blk * L + j0) * es;
    cx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[r * ms];
    const int e = j0 * tstep;
    if (DIR > 0 && m > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], conj(roots[r * e]));
    }
    Dft<T, R, DIR>::run(v);
    if (DIR < 0 && m > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], roots[r * e]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) p[r * ms] = v[r];
  }
}

template <typename T, int DIR>
HD void ip_stage(cx<T>* buf, int ncols, unsigned mcols, int cs, int es, const FftPlan& p, int s, const cx<T>* roots,
                 int tid, int nthr) {
  constexpr int RM = FftMaxRadix<T>::value;
  const int n = p.n, L = p.L[s];
  const unsigned mm = p.m_magic[s];
#define OFDFT_IP_CASE(r)                                                                          \
  case r:                                                                                         \
    if constexpr (r <= RM) ip_stage_r<T, r, DIR>(buf, ncols, mcols, cs, es, n, L, mm, roots, tid, nthr); \
    break;
  switch (p.R[s]) {
    OFDFT_IP_CASE(2)
    OFDFT_IP_CASE(3)
    OFDFT_IP_CASE(4)
    OFDFT_IP_CASE(5)
    OFDFT_IP_CASE(6)
    OFDFT_IP_CASE(7)
    OFDFT_IP_CASE(8)
    OFDFT_IP_CASE(9)
    OFDFT_IP_CASE(10)
    OFDFT_IP_CASE(12)
    OFDFT_IP_CASE(14)
    OFDFT_IP_CASE(15)
    OFDFT_IP_CASE(16)
    default: break;
  }
#undef OFDFT_IP_CASE
}

// One stage whose inputs come from src.ld(c, i) and whose outputs go to
// dst.st(c, i, v) (column c, position i), with the butterfly work split of
// ip_stage_r: a first forward stage can load straight from global memory, a
// last inverse stage store straight to it.
template <typename T, int R, int DIR, class Src, class Dst>
HD void ip_stage_io(const Src& src, const Dst& dst, int ncols, unsigned mcols, int n, int L, unsigned mm,
                    const cx<T>* __restrict__ roots, int tid, int nthr) {
  const int m = L / R;
  const int total = (n / R) * ncols;
  const int tstep = n / L;
  for (int w = tid; w < total; w += nthr) {
    const int bf = magic_div32(w, mcols), c = w - bf * ncols;
    const int blk = magic_div32(bf, mm), j0 = bf - blk * m;
    const int base = blk * L + j0;
    cx<T> v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src.ld(c, base + r * m);
    const int e = j0 * tstep;
    if (DIR > 0 && m > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], conj(roots[r * e]));
    }
    Dft<T, R, DIR>::run(v);
    if (DIR < 0 && m > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], roots[r * e]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) dst.st(c, base + r * m, v[r]);
  }
}

// Stage s of plan p through accessors (a switch over the radix).
template <typename T, int DIR, class Src, class Dst>
HD void ip_stage_acc(const Src& src, const Dst& dst, int ncols, unsigned mcols, const FftPlan& p, int s,
                     const cx<T>* roots, int tid, int nthr) {
  constexpr int RM = FftMaxRadix<T>::value;
  const int n = p.n, L = p.L[s];
  const unsigned mm = p.m_magic[s];
#define OFDFT_IO_CASE(r)                                                                              \
  case r:                                                                                             \
    if constexpr (r <= RM) ip_stage_io<T, r, DIR>(src, dst, ncols, mcols, n, L, mm, roots, tid, nthr); \
    break;
  switch (p.R[s]) {
    OFDFT_IO_CASE(2)
    OFDFT_IO_CASE(3)
    OFDFT_IO_CASE(4)
    OFDFT_IO_CASE(5)
    OFDFT_IO_CASE(6)
    OFDFT_IO_CASE(7)
    OFDFT_IO_CASE(8)
    OFDFT_IO_CASE(9)
    OFDFT_IO_CASE(10)
    OFDFT_IO_CASE(12)
    OFDFT_IO_CASE(14)
    OFDFT_IO_CASE(15)
    OFDFT_IO_CASE(16)
    default: break;
  }
#undef OFDFT_IO_CASE
}

template <typename T, class Op>
HD void ip_stage_op(cx<T>* buf, int ncols, unsigned mcols, int cs, int es, const FftPlan& p, const Op& op, int tid,
                    int nthr) {
  constexpr int RM = FftMaxRadix<T>::value;
  const int n = p.n;
#define OFDFT_OP_CASE(r)                                                                  \
  case r:                                                                                 \
    if constexpr (r <= RM) ip_stage_op_r<T, r>(buf, ncols, mcols, cs, es, n, op, tid, nthr); \
    break;
  switch (p.R[p.nst - 1]) {
    OFDFT_OP_CASE(2)
    OFDFT_OP_CASE(3)
    OFDFT_OP_CASE(4)
    OFDFT_OP_CASE(5)
    OFDFT_OP_CASE(6)
    OFDFT_OP_CASE(7)
    OFDFT_OP_CASE(8)
    OFDFT_OP_CASE(9)
    OFDFT_OP_CASE(10)
    OFDFT_OP_CASE(12)
    OFDFT_OP_CASE(14)
    OFDFT_OP_CASE(15)
    OFDFT_OP_CASE(16)
    default: break;
  }
#undef OFDFT_OP_CASE
}

// Full in-place transform of ncols columns (element i of column c at
// buf[c*cs + i*es]).  DIR = -1: forward, natural -> digit-reversed; DIR = +1:
// inverse, digit-reversed -> natural.  Every thread of the block must call
// it; the data must be complete in shared memory on entry (the caller's
// barrier), and the block synchronises after every stage, so the result is
// complete on return.
template <typename T, int DIR>
HD void fft_inplace(cx<T>* buf, int ncols, int cs, int es, const FftPlan& p, const cx<T>* twtab, int tid, int nthr) {
  const unsigned mcols = magic32(ncols);
  const cx<T>* roots = twtab + p.root;
  if (DIR < 0) {
    for (int s = 0; s < p.nst; ++s) {
      ip_stage<T, -1>(buf, ncols, mcols, cs, es, p, s, roots, tid, nthr);
      BLOCK_SYNC();
    }
  } else {
    for (int s = p.nst - 1; s >= 0; --s) {
      ip_stage<T, 1>(buf, ncols, mcols, cs, es, p, s, roots, tid, nthr);
      BLOCK_SYNC();
    }
  }
}

}  // namespace f32
}  // namespace ofdft
