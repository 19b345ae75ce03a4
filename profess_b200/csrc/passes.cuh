// The FP64 passes of one potential evaluation (CalculatePotentialPlus); the FP32
// slots' passes are those of f32/passes.cuh.
//
// Spectrum layout: field f of a slot is a half spectrum of k1 = n1/2 + 1
// planes, kx-major: element (kx, row j = y + n2 z) at spec[f*Nc + kx*nrows +
// j], so that every (y, z) plane of one kx is contiguous.  Between the
// forward and the inverse transforms along y and z the plane is in the
// digit-reversed order of the in-place FFT (position q holds frequency
// perm[q]); the kernel planes are stored in that order.
//
//   pass 1  X forward : prologue (phi_in, rho and the functional's fields) and
//                       the x-direction real-to-complex FFT of row pairs,
//                       stored kx-major
//   pass YZ           : one (y, z) plane of one field in shared memory:
//                       forward FFT along y and z, the k-space operator
//                       (Hartree 4pi/G^2, vW G^2, the WT kernel, with the 1/N
//                       forward scaling), inverse FFT along z and y
//                       (the three planes of a WGC group together)
//   (planes that do not fit shared memory and the set-up modes run the same
//    work as three passes: Y forward, Z with the operator, Y inverse)
//   pass 5  X inverse : complex-to-real FFT of all fields of a row pair and the
//                       real-space epilogue (potential, chain rule, energies and
//                       the optimiser's fused sums)
//
// Row split (n3 even): the x passes do the radix-2 stage of the z transform,
// on real values (the sums and differences of rows n3/2 apart), and multiply
// its twiddles onto the spectra that they hold in registers anyway.  What is
// left of a plane's z transform is two independent transforms of length n3/2,
// on the contiguous halves z < n3/2 and z >= n3/2 of the plane, so a task of
// the fused y-z pass holds half a plane: twice as many blocks fit an SM (FP64
// 96^2: one block of 149 KB -> three of 75 KB, 411 -> 335 us for 16 cells),
// and planes up to twice the size stay on the fused path (FP64 120^2).
//
// Every block processes one task.  The block functions are force-inlined into
// their kernels: each kernel calls one, and a non-inlined call puts the
// functions' small structs and arrays in local memory.  Blocks of the vector kernel and of pass 5
// store their per-channel sums in the slot's partials; a controller kernel
// that follows (one block per slot) reduces them in a fixed order (the result
// does not depend on block scheduling) and runs the NTN controller.
#pragma once
#include "fft.cuh"
#include "pass_common.cuh"

namespace ofdft {

// Pitch of the x passes' transform buffer: element i of column c at
// buf[i * pitch + c].  Odd, so that threads walking x (a stride of one pitch)
// as well as threads walking the columns touch distinct banks.
HD int x_pitch(int cols) { return cols | 1; }
// Shared memory of an x-forward task with nfb fields (or ion species) and nb
// columns each.
HD size_t xfwd_smem(int n1, int nfb, int nb, size_t esz) { return (size_t)x_pitch(nfb * nb) * n1 * 2 * esz; }
// Shared memory of an x-inverse task with nfb transformed fields (or ion
// species) and nb columns each: the transform buffer, then the reduction scratch.
HD size_t xinv_buf(int n1, int nfb, int nb, size_t esz) { return align16((size_t)x_pitch(nfb * nb) * n1 * 2 * esz); }
HD size_t xinv_smem(int n1, int nfb, int nb, size_t esz) {
  return xinv_buf(n1, nfb, nb, esz) + NCH * 33 * sizeof(double);
}

// phi_in at a point, in one fixed rounding: the x-forward pass (whose fields
// the gradient is taken of) and the x-inverse pass (which stores phi_in as the
// line search's trial) must agree to the last bit, since the finite-difference
// Hessian products divide gradient differences by a small step.
template <typename T>
HD T phi_in(T ca, T a, T cb, T b) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(ca, a, __dmul_rn(cb, b));
#else
  return ca * a + cb * b;
#endif
}

// ------------------------------------------------------------ pass 1
// The x passes keep the packed row pairs of a task in shared memory (row j0
// in the real, row j0 + 1 in the imaginary part).  The forward pass splits the
// two rows' spectra in the registers of its last stage and stores them: one
// round trip through shared memory and its index arithmetic less.
//
// The last forward stage (stride 1) leaves the frequencies kb + M r, r < R,
// M = n / R, in the block whose first element is kb.  The split of the two
// real rows needs Z[k] and Z[n - k], and n - k = (M - kb) + M (R - 1 - r): a
// work item takes the blocks kb and M - kb together and finds every partner
// in its own registers.  The self-paired blocks 0 and (M even) M / 2 are one
// item.  Work items have the row pairs fastest: the pairs of a task are
// adjacent in the kx-major spectra.
HD int x_block_items(int M) { return (M + 1) / 2; }

// Work item (f, p, b) of a last-stage loop over nf fields, the items p of a
// column and nb row pairs.
struct XItem {
  int f, p, b;
};
HD XItem x_item(int w, int nb, unsigned mnb, int np, unsigned mnp) {
  XItem it;
  const int rest = magic_div32(w, mnb);
  it.b = w - rest * nb;
  it.f = magic_div32(rest, mnp);
  it.p = rest - it.f * np;
  return it;
}

// The units of the x passes.  Without the row split a unit is one packed pair
// of adjacent rows (2 u, 2 u + 1).  With it (zs = 2) a unit is the pair in the
// half z < n3/2 and the pair n3/2 further, whose sums and differences take the
// pairs' places in the x transforms (the radix-2 z stage, on real values),
// so that a unit has zs columns: 0 the sums, 1 the differences.  A shift of
// the cell by n3/2 exchanges the two pairs and with that only the sign of
// column 1: densities with that symmetry keep it to the last bit.
struct RowMap {
  int zs, half, n2, nrows;  // half: rows of a half, n2 * zh
  HD int row(int u, int col) const { return 2 * u + col * half; }  // first row of the pair
  HD bool has1(int u) const { return 2 * u + 1 < half; }
};
HD RowMap row_map(const SlotDev& s) { return RowMap{s.zs, s.n2 * s.zh, s.n2, s.n2 * s.n3}; }

// A column's pair in the (y, z) planes of the spectra: its first row, whether
// it has a second one, and (column 1) the twiddles W_{n3}^z of its rows' radix-2 z stage.
template <typename T>
struct PairIO {
  int row;
  bool has1, tw;
  cx<T> wa, wb;
};
template <typename T>
HD PairIO<T> pair_io(const RowMap& rm, int u, int col, const cx<T>* __restrict__ wz) {
  PairIO<T> p;
  p.row = rm.row(u, col);
  p.has1 = rm.has1(u);
  p.tw = col != 0;
  p.wa = p.wb = mk<T>(T(1), T(0));
  if (p.tw) {
    p.wa = wz[2 * u / rm.n2];
    p.wb = p.has1 ? wz[(2 * u + 1) / rm.n2] : p.wa;
  }
  return p;
}

// The spectra of the two real rows of Z = A + i B from z = Z[k] and zn = Z[n -
// k], A = (z + conj zn) / 2 and B = (z - conj zn) / 2i, times the z twiddles.
template <typename T, bool TW>
HD void x_store(cx<T>* __restrict__ o, cx<T> z, cx<T> zn, const PairIO<T>& io) {
  cx<T> a = mk<T>((z.x + zn.x) * T(0.5), (z.y - zn.y) * T(0.5));
  cx<T> b = mk<T>((z.y + zn.y) * T(0.5), (zn.x - z.x) * T(0.5));
  if (TW) {
    a = cmul(a, io.wa);
    b = cmul(b, io.wb);
  }
  o[0] = a;
  if (io.has1) o[1] = b;
}
// The loads' mirror: the two rows' values (a, b) of frequency k, and the
// packed sequence Z = A + i B at k and n - k in their place.
template <typename T>
HD void x_load(const cx<T>* __restrict__ o, const PairIO<T>& io, cx<T>& a, cx<T>& b) {
  a = o[0];
  b = io.has1 ? o[1] : mk<T>(T(0), T(0));
}
template <typename T>
HD void x_untwiddle(cx<T>& a, cx<T>& b, const PairIO<T>& io) {
  a = cmul(a, conj(io.wa));
  b = cmul(b, conj(io.wb));
}
template <typename T>
HD void x_pack(cx<T>& a, cx<T>& b) {
  const cx<T> A = a, B = b;
  a = mk<T>(A.x - B.y, A.y + B.x);
  b = mk<T>(A.x + B.y, B.x - A.y);
}

// The outputs of blocks va (frequencies from oa on) and vb (from ob on).
template <typename T, int R, bool TW>
HD void x_store_blocks(cx<T>* __restrict__ oa, cx<T>* __restrict__ ob, size_t rs, const cx<T>* va, const cx<T>* vb,
                       bool first, bool even, const PairIO<T>& io) {
  if (first) {
#pragma unroll
    for (int r = 0; r <= R / 2; ++r) x_store<T, TW>(oa + r * rs, va[r], va[(R - r) % R], io);
    if (even) {
#pragma unroll
      for (int r = 0; r < (R + 1) / 2; ++r) x_store<T, TW>(ob + r * rs, vb[r], vb[R - 1 - r], io);
    }
  } else {
#pragma unroll
    for (int r = 0; r < (R + 1) / 2; ++r) x_store<T, TW>(oa + r * rs, va[r], vb[R - 1 - r], io);
#pragma unroll
    for (int r = 0; r < R / 2; ++r) x_store<T, TW>(ob + r * rs, vb[r], va[R - 1 - r], io);
  }
}

// The last forward stage (radix R, no twiddles) of nf * nc columns (nc = zs *
// nb, nb units), the split and the stores.  ip: position of frequency k after
// the forward transform.
template <typename T, int R>
HD void x_last_split_r(const cx<T>* __restrict__ buf, cx<T>* __restrict__ spec, long long Nc, const RowMap& rm, int u0,
                       int nf, int nb, int es, int M, const int* __restrict__ ip, const cx<T>* __restrict__ wz,
                       int tid, int nthr) {
  const int np = x_block_items(M), nc = rm.zs * nb;
  const unsigned mnc = magic32(nc), mnp = magic32(np);
  for (int w = tid; w < nf * np * nc; w += nthr) {
    const XItem it = x_item(w, nc, mnc, np, mnp);
    const int kb = it.p, kq = kb == 0 ? ((M & 1) ? 0 : M / 2) : M - kb;
    const cx<T>* c = buf + it.f * nc + it.b;
    const cx<T>* pa = c + ip[kb] * es;
    const cx<T>* pb = c + ip[kq] * es;
    cx<T> va[R], vb[R];
#pragma unroll
    for (int r = 0; r < R; ++r) va[r] = pa[r * es];
#pragma unroll
    for (int r = 0; r < R; ++r) vb[r] = pb[r * es];
    Dft<T, R, -1>::run(va);
    Dft<T, R, -1>::run(vb);
    const int col = it.b >= nb ? 1 : 0;
    const PairIO<T> io = pair_io<T>(rm, u0 + it.b - col * nb, col, wz);
    cx<T>* o = spec + (size_t)it.f * (size_t)Nc + io.row;
    const size_t rs = (size_t)M * rm.nrows;
    const size_t da = (size_t)kb * rm.nrows, db = (size_t)kq * rm.nrows;
    if (io.tw) x_store_blocks<T, R, true>(o + da, o + db, rs, va, vb, kb == 0, (M & 1) == 0, io);
    else x_store_blocks<T, R, false>(o + da, o + db, rs, va, vb, kb == 0, (M & 1) == 0, io);
  }
}

template <typename T>
HD void x_last_split(const cx<T>* buf, cx<T>* spec, long long Nc, const RowMap& rm, int u0, int nf, int nb, int es,
                     const StagePlan& p, const int* ip, const cx<T>* wz, int tid, int nthr) {
  const int R = p.R[p.nst - 1], M = p.n / R;
#define OFDFT_LAST_CASE(r)                                                               \
  case r:                                                                                \
    x_last_split_r<T, r>(buf, spec, Nc, rm, u0, nf, nb, es, M, ip, wz, tid, nthr); \
    break;
  static_assert(XLAST_MAX == 4, "the radices below");
  switch (R) {
    OFDFT_LAST_CASE(1)
    OFDFT_LAST_CASE(2)
    OFDFT_LAST_CASE(3)
    OFDFT_LAST_CASE(4)
    default: break;
  }
#undef OFDFT_LAST_CASE
}

// Sum and difference with one rounding each: never contracted with the
// operands' own products, so that exchanging a and b changes only a sign.
template <typename T>
HD T add_rn(T a, T b) {
#if defined(__CUDA_ARCH__)
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}

// The gather of an inverse task: the packed sequences Z = A + i B of every
// unit's row pairs at the digit-reversed positions that the inverse transform
// takes, Z[k] from the stored k <= n/2 and Z[n - k] from its conjugate
// symmetry (a self-paired k, 0 and n/2, takes the real parts only, as c2r
// does).  With the row split the inverse radix-2 z stage gives the spectra of
// the rows z and z + n3/2: a unit's columns are its two pairs from here on.
// Consecutive threads read consecutive units of one kx.
template <typename T>
HD void x_gather(cx<T>* __restrict__ buf, const cx<T>* __restrict__ spec, long long Nc, const RowMap& rm, int u0,
                 int nf, int nb, int es, const StagePlan& p, const int* __restrict__ ip, const cx<T>* __restrict__ wz,
                 int tid, int nthr) {
  const int n = p.n, k1 = n / 2 + 1, nc = rm.zs * nb;
  const unsigned mnb = magic32(nb), mk1 = magic32(k1);
#pragma unroll 2
  for (int w = tid; w < nf * k1 * nb; w += nthr) {
    const XItem it = x_item(w, nb, mnb, k1, mk1);
    const int k = it.p;
    const bool self = k == 0 || 2 * k == n;
    PairIO<T> io = pair_io<T>(rm, u0 + it.b, 0, wz);
    const cx<T>* o = spec + (size_t)it.f * (size_t)Nc + (size_t)k * rm.nrows;
    cx<T> a, b, c = mk<T>(T(0), T(0)), d = c;
    x_load(o + io.row, io, a, b);
    if (rm.zs == 2) {
      io = pair_io<T>(rm, u0 + it.b, 1, wz);
      x_load(o + io.row, io, c, d);
      x_untwiddle(c, d, io);
    }
    cx<T>* q = buf + it.f * nc + it.b;
    cx<T>* qk = q + ip[k] * es;
    cx<T>* qn = q + ip[self ? k : n - k] * es;
    for (int col = 0; col < rm.zs; ++col) {
      cx<T> A = mk<T>(add_rn(a.x, c.x), add_rn(a.y, c.y)), B = mk<T>(add_rn(b.x, d.x), add_rn(b.y, d.y));
      if (self) {
        *qk = mk<T>(A.x, B.x);
      } else {
        x_pack(A, B);
        *qk = A;
        *qn = B;
      }
      qk += nb;
      qn += nb;
      c = mk<T>(-c.x, -c.y);
      d = mk<T>(-d.x, -d.y);
    }
  }
}

// rho and sqrt(rho) of an input value (phi_in, or rho itself in rho mode).
template <typename T> HD T in_rho(T x, int rho_mode) { return rho_mode ? x : x * x; }
template <typename T> HD T in_sqrt(T x, int rho_mode) { return rho_mode ? m_sqrt(x) : (x < T(0) ? -x : x); }
// rho^(5/6) = a^2 a^(-1/3) of rho and a = sqrt(rho) (out: a is outside
// m_icbrt's range).
template <typename T>
HD T pow56(T rho, T a, bool& out) {
  out = out || icbrt_out(a);
  return rho * m_icbrt(a);
}

// All forward fields of NP points from their evaluation inputs (WT: rho,
// rho^beta, sqrt(rho) - shift and, when alpha != beta, rho^alpha; WGC: rho, sqrt(rho) - shift,
// then for x = alpha and x = beta: rho^x, theta rho^x, theta^2 rho^x / 2 with
// theta = rho - rho*), with each power computed once per point: put(f, v) for
// every field.  POW56: the WT functional with both exponents 5/6 (its fall-back
// power is a call).  Every index is a constant: arrays indexed in a loop go to
// local memory.
template <typename T, int KS, bool POW56, int NP, class Put>
HD void point_fields(const FieldPar<T>& fp, int rho_mode, int nf, T shift, const T* x, Put put) {
  T rho[NP], sq[NP], v[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    rho[k] = in_rho(x[k], rho_mode);
    sq[k] = in_sqrt(x[k], rho_mode);
  }
  put(0, rho);
#pragma unroll
  for (int k = 0; k < NP; ++k) v[k] = sq[k] - shift;
  put(KS == KS_WT ? 2 : 1, v);
  if constexpr (KS == KS_WT) {
    if constexpr (POW56) {
      bool slow = false;
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = pow56(rho[k], sq[k], slow);
      if (slow) {
#pragma unroll
        for (int k = 0; k < NP; ++k) v[k] = m_pow_call(rho[k], fp.beta);
      }
      put(1, v);
    } else {
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = m_pow(rho[k], fp.beta);
      put(1, v);
      if (nf > 3) {
#pragma unroll
        for (int k = 0; k < NP; ++k) v[k] = m_pow(rho[k], fp.alpha);
        put(3, v);
      }
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = m_pow(rho[k], h == 0 ? fp.alpha : fp.beta);
      put(2 + 3 * h, v);
      T u[NP];
#pragma unroll
      for (int k = 0; k < NP; ++k) u[k] = (rho[k] - fp.rho_s) * v[k];
      put(3 + 3 * h, u);
#pragma unroll
      for (int k = 0; k < NP; ++k) u[k] = (rho[k] - fp.rho_s) * (rho[k] - fp.rho_s) * v[k] / T(2);
      put(4 + 3 * h, u);
    }
  }
}

// The constant that sqrt(rho) is transformed without: the mean of sqrt(rho) at
// 32 points spread over the cell (a lane's share each; every warp has the same
// sum).  The von Weizsaecker term takes the Laplacian of sqrt(rho), which a
// constant is not in, and multiplies the transform's rounding errors, which
// are of the size of what is transformed, by up to the largest |G|^2: they
// are most of the error of a potential (RMS over the potential's, 96^3: 2.7e-14
// with sqrt(rho) whole, 1.0e-14 so; 3 us of 230 of the pass for 16 cells, 26 with
// eight points that every thread reads).
template <typename T>
HD T vw_shift(const EvalIn<T>& in, const SlotDev& s, int tid) {
  auto at = [&](int k) {
    const int i = (((k * s.n3) >> 5) * s.n2 + (((k * 7 & 31) * s.n2) >> 5)) * s.n1 + (((k * 11 & 31) * s.n1) >> 5);
    T x = in.A[i];
    if (!in.rho_mode) x = in.cb != T(0) ? in.ca * x + in.cb * in.B[i] : in.ca * x;
    return in_sqrt(x, in.rho_mode);
  };
#if defined(__CUDA_ARCH__)
  T sum = at(tid & 31);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#else
  (void)tid;
  T sum = T(0);
  for (int k = 0; k < 32; ++k) sum += at(k);
#endif
  return sum * T(1.0 / 32.0);
}

template <int N> struct Count { static constexpr int value = N; };

// Every field of a range of units in one block: element i of column f*nc +
// col*nb + b at buf[i*es + f*nc + col*nb + b].
template <typename T, int KS>
HD void xfwd_block(const Args<T>& a, int bid, int tid, int nthr, char* smem) {
  const Task t = a.tasks[bid];
  const SlotDev& s = a.slots[t.slot];
  const Ctl& c = a.ctl[t.slot];
  if (c.status != ST_RUNNING || c.ev == EV_NONE) return;
  const int u0 = t.b, nb = t.c;
  const int ev = c.ev;
  const bool setup = ev == EV_ION || ev == EV_FORCE;  // one field: the inputs as they are
  const int nf = ev == EV_ION ? s.ion.nspec : ev == EV_FORCE ? 1 : s.nf;
  const int n1 = s.n1, zs = s.zs, nc = zs * nb;
  const RowMap rm = row_map(s);
  const int es = x_pitch(nf * nc);
  const StagePlan& px = s.qxf;
  cx<T>* buf = (cx<T>*)smem;
  const EvalIn<T> in = eval_in<T>(s, c);
  const FieldPar<T> fp = field_par<T>(s);
  const T shift = setup ? T(0) : vw_shift(in, s, tid);
  const unsigned mn1 = magic32(n1);
  const bool two = !in.rho_mode && in.cb != T(0);
  // the inputs of NP points at once: every load of both arrays first.  A
  // missing second row has the first one's inputs (valid ones: the functional's
  // powers of a zero density may be infinite), and put stores zero fields for it.
  auto inputs = [&](auto np, const T* __restrict__ A, const int* idx, T* x) {
    constexpr int NP = decltype(np)::value;
#pragma unroll
    for (int k = 0; k < NP; ++k) x[k] = A[idx[k]];
    if (ev != EV_ION && !in.rho_mode) {
      if (two) {
        T y[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) y[k] = in.B[idx[k]];
#pragma unroll
        for (int k = 0; k < NP; ++k) x[k] = phi_in(in.ca, x[k], in.cb, y[k]);
      } else {
#pragma unroll
        for (int k = 0; k < NP; ++k) x[k] *= in.ca;
      }
      if (ev == EV_FORCE) {
#pragma unroll
        for (int k = 0; k < NP; ++k) x[k] *= x[k];
      }
    }
  };
  if (!setup && (KS == KS_WGC || !fp.pow56)) {
    // General powers: a work item is one row of a pair (and its partner n3/2
    // further), so that twice as many threads each compute half as many powers
    // one after the other (8 x 64^3, unequal exponents: 118 us of the pass with
    // the pair as the item, its powers in loops over local memory, and a last
    // stage of radix 8; 89 us so).  Consecutive threads take the two rows of a
    // pair: their fields are the two parts of one complex value.
    for (int w = tid; w < 2 * nb * n1; w += nthr) {
      const int p = w & 1, b = magic_div32(w >> 1, mn1), i = (w >> 1) - b * n1;
      const bool has = p == 0 || rm.has1(u0 + b);
      const int i0 = (rm.row(u0 + b, 0) + (has ? p : 0)) * n1 + i;
      T* d = (T*)(buf + i * es + b) + p;
      if (zs == 1) {
        const int idx[1] = {i0};
        T x[1];
        inputs(Count<1>(), in.A, idx, x);
        point_fields<T, KS, false, 1>(fp, in.rho_mode, nf, shift, x,
                                      [&](int f, const T* v) { d[2 * (f * nc)] = has ? v[0] : T(0); });
      } else {
        const int idx[2] = {i0, i0 + rm.half * n1};
        T x[2];
        inputs(Count<2>(), in.A, idx, x);
        point_fields<T, KS, false, 2>(fp, in.rho_mode, nf, shift, x, [&](int f, const T* v) {
          d[2 * (f * nc)] = has ? add_rn(v[0], v[1]) : T(0);
          d[2 * (f * nc + nb)] = has ? add_rn(v[0], -v[1]) : T(0);
        });
      }
    }
  } else {
    for (int f0 = 0; f0 < (ev == EV_ION ? nf : 1); ++f0) {
      const T* __restrict__ A = ev == EV_ION ? (const T*)s.buf[B_PHI + f0] : in.A;
#pragma unroll 2
      for (int w = tid; w < nb * n1; w += nthr) {
        const int b = magic_div32(w, mn1), i = w - b * n1;
        const bool has1 = rm.has1(u0 + b);
        const int i0 = rm.row(u0 + b, 0) * n1 + i, i1 = has1 ? i0 + n1 : i0;
        cx<T>* d = buf + i * es + b;
        if (zs == 1) {
          const int idx[2] = {i0, i1};
          T x[2];
          inputs(Count<2>(), A, idx, x);
          auto put = [&](int f, const T* v) { d[f * nc] = mk<T>(v[0], has1 ? v[1] : T(0)); };
          if (setup) put(f0, x);
          else if constexpr (KS == KS_WT) point_fields<T, KS, true, 2>(fp, in.rho_mode, nf, shift, x, put);
        } else {
          const int hs = rm.half * n1;
          const int idx[4] = {i0, i1, i0 + hs, i1 + hs};
          T x[4];
          inputs(Count<4>(), A, idx, x);
          auto put = [&](int f, const T* v) {
            d[f * nc] = mk<T>(add_rn(v[0], v[2]), has1 ? add_rn(v[1], v[3]) : T(0));
            d[f * nc + nb] = mk<T>(add_rn(v[0], -v[2]), has1 ? add_rn(v[1], -v[3]) : T(0));
          };
          if (setup) put(f0, x);
          else if constexpr (KS == KS_WT) point_fields<T, KS, true, 4>(fp, in.rho_mode, nf, shift, x, put);
        }
      }
    }
  }
  BLOCK_SYNC();
  const unsigned mcols = magic32(nf * nc);
  for (int st = 0; st < px.nst - 1; ++st) {
    ip_stage<T, -1>(buf, nf * nc, mcols, 1, es, px, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  x_last_split<T>(buf, (cx<T>*)s.spec, s.Nc, rm, u0, nf, nb, es, px, a.idx + px.iperm, a.tw + s.qz.root, tid, nthr);
}

// The operator of one z-pass tile of a set-up mode (G_ION, G_FORCE): res[i*NB
// + q*nb + b] holds species q at z position z0 + i (frequency kz = permz[z0 +
// i]) and y position y0 + b (ky = permy[y0 + b]), for kx; the results replace
// the inputs.
template <typename T>
HD void zpass_setup(const SlotDev& s, int kind, int gn, cx<T>* res, int NB, int nb, int kx, int y0, int z0,
                    const int* __restrict__ permy, const int* __restrict__ permz, int tid, int nthr) {
  const int n2 = s.n2, n3 = s.n3;
  const unsigned mnb = magic32(nb);
  for (int w = tid; w < nb * s.zh; w += nthr) {
    const int i = magic_div32(w, mnb), b = w - i * nb;
    const int ky = permy[y0 + b], kz = permz[z0 + i];
    const int m2 = signed_freq(ky, n2), m3 = signed_freq(kz, n3);
    cx<T>* e = res + i * NB + b;
    const double gx = s.recip[0] * kx + s.recip[3] * m2 + s.recip[6] * m3;
    const double gy = s.recip[1] * kx + s.recip[4] * m2 + s.recip[7] * m3;
    const double gz = s.recip[2] * kx + s.recip[5] * m2 + s.recip[8] * m3;
    const double q = sqrt(gx * gx + gy * gy + gz * gz);
    switch (kind) {
      case G_ION: {  // conj(sum_s V_s(|G|) b1 b2 b3 S_s) N / vol, times the 1/N forward scale
        // (IonElectronPotRecipSpline, IonElectronSpline.f90:180-203)
        const cx<double> bb = cmul(cmul(s.ion.b1[kx], s.ion.b2[ky]), s.ion.b3[kz]);
        double yr = 0.0, yi = 0.0;
        for (int sp = 0; sp < gn; ++sp) {
          const double v = psp_value(s.ion, sp, q);
          const cx<T> F = e[sp * nb];
          yr += v * (double)F.x;
          yi += v * (double)F.y;
        }
        const double pr = yr * bb.x - yi * bb.y, pim = yr * bb.y + yi * bb.x;
        e[0] = mk<T>((T)(pr / s.vol), (T)(-pim / s.vol));
        break;
      }
      default: {  // G_FORCE: rho(G) V_s(|G|) b1 b2 b3 per species, G = 0 excluded
        // (IonElectronForcesSpline, IonElectronSpline.f90:300-330)
        const cx<double> bb = cmul(cmul(s.ion.b1[kx], s.ion.b2[ky]), s.ion.b3[kz]);
        const cx<T> F = e[0];
        const bool g0 = kx == 0 && ky == 0 && kz == 0;
        for (int sp = gn - 1; sp >= 0; --sp) {
          const double v = g0 ? 0.0 : psp_value(s.ion, sp, q) * s.inv_n;
          const double fr = (double)F.x * v, fi = (double)F.y * v;
          e[sp * nb] = mk<T>((T)(fr * bb.x - fi * bb.y), (T)(fr * bb.y + fi * bb.x));
        }
        break;
      }
    }
  }
}

// The last forward stage (radix R, stride 1) of the three columns of a WGC
// group, the second-order WGC operator (KEDF_WGC.f90:219-236) and the first
// inverse stage, in registers.  Field p of column c, position i: buf[c*cs +
// i*es + p*ps]; the kernel planes K1..K4 there: kern[j*Nc + c*kc + i*ki].
// The kernel values of a butterfly are loaded one position at a time.
template <typename T, int R>
HD void ip_stage_wgc3_r(cx<T>* __restrict__ buf, int ncols, unsigned mcols, int cs, int es, int ps, int n,
                        const T* __restrict__ kern, int kc, int ki, long long Nc, T sc, int tid, int nthr) {
  const int total = (n / R) * ncols;
  for (int w = tid; w < total; w += nthr) {
    const int blk = magic_div32(w, mcols), c = w - blk * ncols;
    cx<T>* p0 = buf + c * cs + blk * R * es;
    cx<T> v0[R], v1[R], v2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      v0[r] = p0[r * es];
      v1[r] = p0[r * es + ps];
      v2[r] = p0[r * es + 2 * ps];
    }
    Dft<T, R, -1>::run(v0);
    Dft<T, R, -1>::run(v1);
    Dft<T, R, -1>::run(v2);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int kidx = c * kc + (blk * R + r) * ki;
      const T K1 = kern[kidx], K2 = kern[Nc + kidx], K3 = kern[2 * Nc + kidx], K4 = kern[3 * Nc + kidx];
      const cx<T> F0 = v0[r], F1 = v1[r], F2 = v2[r];
      v0[r] = (F0 * K1 + F1 * K2 + F2 * K3) * sc;
      v1[r] = (F0 * K2 + F1 * K4) * sc;
      v2[r] = F0 * (K3 * sc);
    }
    Dft<T, R, 1>::run(v0);
    Dft<T, R, 1>::run(v1);
    Dft<T, R, 1>::run(v2);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      p0[r * es] = v0[r];
      p0[r * es + ps] = v1[r];
      p0[r * es + 2 * ps] = v2[r];
    }
  }
}

template <typename T>
HD void ip_stage_wgc3(cx<T>* buf, int ncols, unsigned mcols, int cs, int es, int ps, const StagePlan& p, const T* kern,
                      int kc, int ki, long long Nc, T sc, int tid, int nthr) {
  const int n = p.n;
#define OFDFT_RADIX_DO(r) \
  ip_stage_wgc3_r<T, r>(buf, ncols, mcols, cs, es, ps, n, kern, kc, ki, Nc, sc, tid, nthr)
  OFDFT_RADIX_SWITCH(p.R[p.nst - 1])
#undef OFDFT_RADIX_DO
}

// The Hartree / vW factor at (column z, y position q) of the fused pass.
template <typename T>
struct GOp {
  GFactor<T> gf;
  int kind, kx, n2, n3;  // n3: the whole axis
  const int* __restrict__ permy;
  const int* __restrict__ permz;  // of the task's first z position
  HD T operator()(int z, int q) const {
    return gf(kind, kx, signed_freq(permy[q], n2), signed_freq(permz[z], n3));
  }
};

// ------------------------------------------------------------ Y passes (split path)
// Task (field f, kx, z tile): nz columns of n2 contiguous values (one per
// z), transformed along y in place: forward (dir < 0) natural -> digit
// reversed, inverse (dir > 0) back.
template <typename T>
HD void ypass_block(const Args<T>& a, int bid, int tid, int nthr, char* smem, int dir) {
  const Task t = a.tasks[bid];
  const SlotDev& s = a.slots[t.slot];
  const Ctl& c = a.ctl[t.slot];
  if (c.status != ST_RUNNING || c.ev == EV_NONE) return;
  const int f = t.a, kx = t.b, z0 = tile_first(t.c), nz = tile_width(t.c);
  if (c.ev == EV_ION && f >= (dir < 0 ? s.ion.nspec : 1)) return;
  if (c.ev == EV_FORCE && f >= (dir < 0 ? 1 : s.ion.nspec)) return;
  if (c.ev == EV_STRESS && dir > 0) return;  // forward spectra only
  const int n2 = s.n2, P = odd_pitch(n2);
  cx<T>* buf = (cx<T>*)smem;
  cx<T>* __restrict__ sp =
      (cx<T>*)s.spec + (size_t)f * (size_t)s.Nc + (size_t)kx * (n2 * s.n3) + (size_t)z0 * n2;
  const unsigned mn2 = magic32(n2);
#pragma unroll 4
  for (int w = tid; w < nz * n2; w += nthr) {
    const int zc = magic_div32(w, mn2), y = w - zc * n2;
    buf[zc * P + y] = sp[w];
  }
  BLOCK_SYNC();
  if (dir < 0) fft_inplace<T, -1>(buf, nz, P, 1, s.qy, a.tw, tid, nthr);
  else fft_inplace<T, 1>(buf, nz, P, 1, s.qy, a.tw, tid, nthr);
#pragma unroll 4
  for (int w = tid; w < nz * n2; w += nthr) {
    const int zc = magic_div32(w, mn2), y = w - zc * n2;
    sp[w] = buf[zc * P + y];
  }
}

// ------------------------------------------------------------ Z pass (split path)
// A z-pass tile in the spectra: column q*nb + b (field q of the group, y
// position b of the tile), position i.
template <typename T>
struct TileIO {
  cx<T>* base;
  long long Nc;
  int nb, n2;
  unsigned mnb;
  HD size_t at(int c, int i) const {
    const int q = magic_div32(c, mnb), b = c - q * nb;
    return (size_t)q * (size_t)Nc + (size_t)i * n2 + b;
  }
  HD cx<T> ld(int c, int i) const { return base[at(c, i)]; }
  HD void st(int c, int i, cx<T> v) const { base[at(c, i)] = v; }
};
template <typename T>
struct TileKern {  // the WT kernel at (column, position) of a tile, times the 1/N forward scale
  const T* __restrict__ kern;
  T sc;
  int n2;
  HD T operator()(int b, int i) const { return kern[i * n2 + b] * sc; }
};
template <typename T>
struct TileG {  // the Hartree or vW factor there
  GOp<T> g;
  HD T operator()(int b, int i) const { return g(i, b); }
};

// Task (group g, kx and half of the row split, y tile): the group's gn
// fields at ny consecutive y positions, the zh z values of the half, as gn*ny
// columns [z][q*ny + b]: forward FFT along z, the group's operator, inverse
// FFT along z.  As in the fused pass the first forward stage loads straight
// from the spectra, the last forward stage, the operator and the first
// inverse stage run in registers, and the last inverse stage stores straight
// to the spectra: half of the round trips through shared memory of a staged
// tile, generic stages and a separate operator loop (1152 ions, 160 x 160 x
// 256 WGC: 832 -> 338 us).
template <typename T, int KS>
HD void zpass_block(const Args<T>& a, int bid, int tid, int nthr, char* smem) {
  const Task t = a.tasks[bid];
  const SlotDev& s = a.slots[t.slot];
  const Ctl& c = a.ctl[t.slot];
  if (c.status != ST_RUNNING || c.ev == EV_NONE) return;
  const int g = t.a, kx = t.b / s.zs, half = t.b - kx * s.zs, y0 = tile_first(t.c), nb = tile_width(t.c);
  const int ev = c.ev;
  const bool setup_mode = ev == EV_ION || ev == EV_FORCE;
  if (setup_mode && g != 0) return;
  const int n2 = s.n2, zh = s.zh, z0 = half * zh;
  const int kind = ev == EV_ION ? G_ION : ev == EV_FORCE ? G_FORCE : s.group_kind[g];
  const int gn = setup_mode ? s.ion.nspec : s.group_nf[g];
  const int NB = gn * nb;
  const long long Nc = s.Nc;
  const size_t at = (size_t)kx * (n2 * s.n3) + (size_t)z0 * n2 + y0;
  cx<T>* __restrict__ spec = (cx<T>*)s.spec + (size_t)(setup_mode ? 0 : s.group_f0[g]) * (size_t)Nc + at;
  cx<T>* buf = (cx<T>*)smem;
  const StagePlan& pz = s.qzh;
  const unsigned mNB = magic32(NB), mnb = magic32(nb);
  if (setup_mode || ev == EV_STRESS) {
    const int gin = ev == EV_FORCE ? 1 : gn;  // fields loaded
    const int gout = ev == EV_ION ? 1 : gn;   // fields stored
    for (int w = tid; w < NB * zh; w += nthr) {
      const int i = magic_div32(w, mNB), qb = w - i * NB;
      const int q = magic_div32(qb, mnb), b = qb - q * nb;
      buf[w] = q < gin ? spec[(size_t)q * Nc + i * n2 + b] : mk<T>(T(0), T(0));
    }
    BLOCK_SYNC();
    fft_inplace<T, -1>(buf, NB, 1, NB, pz, a.tw, tid, nthr);
    if (setup_mode) {
      zpass_setup<T>(s, kind, gn, buf, NB, nb, kx, y0, z0, a.idx + s.qy.perm, a.idx + s.qz.perm, tid, nthr);
      BLOCK_SYNC();
      fft_inplace<T, 1>(buf, NB, 1, NB, pz, a.tw, tid, nthr);
    }
    for (int w = tid; w < NB * zh; w += nthr) {  // EV_STRESS keeps the forward spectra
      const int i = magic_div32(w, mNB), qb = w - i * NB;
      const int q = magic_div32(qb, mnb), b = qb - q * nb;
      if (q < gout) spec[(size_t)q * Nc + i * n2 + b] = buf[w];
    }
    return;
  }
  const TileIO<T> glob{spec, Nc, nb, n2, mnb};
  const PlaneIO<T> tile{buf, NB};
  if (pz.nst > 1) {
    ip_stage_acc<T, -1>(glob, tile, NB, mNB, pz, 0, a.tw, tid, nthr);
    BLOCK_SYNC();
    for (int st = 1; st < pz.nst - 1; ++st) {
      ip_stage<T, -1>(buf, NB, mNB, 1, NB, pz, st, a.tw, tid, nthr);
      BLOCK_SYNC();
    }
  } else {
    for (int w = tid; w < NB * zh; w += nthr) {
      const int i = magic_div32(w, mNB);
      buf[w] = glob.ld(w - i * NB, i);
    }
    BLOCK_SYNC();
  }
  const T sc = (T)s.inv_n;
  if (kind == G_WGC3) {
    if constexpr (KS == KS_WGC)
      ip_stage_wgc3<T>(buf, nb, mnb, 1, NB, nb, pz, (const T*)s.kern + at, 1, n2, Nc, sc, tid, nthr);
  } else if (kind == G_KMUL) {
    const TileKern<T> op{(const T*)s.kern + at, sc, n2};
    ip_stage_op<T>(buf, nb, mnb, 1, NB, pz, op, tid, nthr);
  } else {
    TileG<T> op;
    op.g.gf.init(s);
    op.g.kind = kind;
    op.g.kx = kx;
    op.g.n2 = n2;
    op.g.n3 = s.n3;
    op.g.permy = a.idx + s.qy.perm + y0;
    op.g.permz = a.idx + s.qz.perm + z0;
    ip_stage_op<T>(buf, nb, mnb, 1, NB, pz, op, tid, nthr);
  }
  BLOCK_SYNC();
  if (pz.nst > 1) {
    for (int st = pz.nst - 2; st >= 1; --st) {
      ip_stage<T, 1>(buf, NB, mNB, 1, NB, pz, st, a.tw, tid, nthr);
      BLOCK_SYNC();
    }
    ip_stage_acc<T, 1>(tile, glob, NB, mNB, pz, 0, a.tw, tid, nthr);
  } else {
    for (int w = tid; w < NB * zh; w += nthr) {
      const int i = magic_div32(w, mNB);
      glob.st(w - i * NB, i, buf[w]);
    }
  }
}

// ------------------------------------------------------------ YZ pass (fused path)
// Task (WGC group g, kx, half): the three fields' (y, z) half planes at kx together in
// shared memory, interleaved along y (field p, y, z at z*P3 + p*n2 + y, P3 =
// odd pitch of 3*n2), since the WGC operator mixes the three at each
// frequency.  The z transforms run over all 3*n2 columns at once, the y
// transforms plane by plane, and the last forward y stage, the operator and
// the first inverse y stage run in registers for the three planes together.
// As the single-field task, one read and one write of each plane in HBM.
template <typename T>
HD void yz_wgc3_block(const Args<T>& a, const SlotDev& s, int g, int kx, int half, cx<T>* buf, int tid, int nthr) {
  const int n2 = s.n2, n3 = s.zh, nc = 3 * n2, P3 = odd_pitch(nc);
  const size_t at = (size_t)kx * (n2 * s.n3) + half * n3 * n2;  // the half's first element in a field's spectra
  const long long Nc = s.Nc;
  const StagePlan& py = s.qy;
  const StagePlan& pz = s.qzh;
  const unsigned mnc = magic32(nc), mn3 = magic32(n3);
  const Planes3IO<T> glob{(cx<T>*)s.spec + (size_t)s.group_f0[g] * (size_t)Nc + at, Nc, n2, magic32(n2)};
  const PlaneIO<T> rows{buf, P3};
  ip_stage_acc<T, -1>(glob, rows, nc, mnc, pz, 0, a.tw, tid, nthr);
  BLOCK_SYNC();
  for (int st = 1; st < pz.nst; ++st) {
    ip_stage<T, -1>(buf, nc, mnc, 1, P3, pz, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  for (int st = 0; st < py.nst - 1; ++st) {
    for (int p = 0; p < 3; ++p) ip_stage<T, -1>(buf + p * n2, n3, mn3, P3, 1, py, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  ip_stage_wgc3<T>(buf, n3, mn3, P3, 1, n2, py, (const T*)s.kern + at, n2, 1, Nc, (T)s.inv_n, tid, nthr);
  BLOCK_SYNC();
  for (int st = py.nst - 2; st >= 0; --st) {
    for (int p = 0; p < 3; ++p) ip_stage<T, 1>(buf + p * n2, n3, mn3, P3, 1, py, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  for (int st = pz.nst - 1; st >= 1; --st) {
    ip_stage<T, 1>(buf, nc, mnc, 1, P3, pz, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  ip_stage_acc<T, 1>(rows, glob, nc, mnc, pz, 0, a.tw, tid, nthr);
}

// Task (group g, kx, half) of a single-field group: half a (y, z) plane of the
// field at kx (n2*zh contiguous values; the whole plane without the row
// split, zh = n3) in shared memory, rows of odd pitch
// P.  The forward FFT along z loads its first stage straight from the
// spectra (consecutive threads, consecutive y); then the forward FFT along y;
// its last stage, the operator and the first inverse stage run in registers
// in one pass; then the inverse along y and z, whose last stage stores
// straight to the spectra.  One read and one write of the plane in HBM.
// KS = KS_WGC also takes the three-field WGC groups (yz_wgc3_block); the WT
// instantiation carries none of their code.
template <typename T, int KS>
HD void yzpass_block(const Args<T>& a, int bid, int tid, int nthr, char* smem) {
  const Task t = a.tasks[bid];
  const SlotDev& s = a.slots[t.slot];
  const Ctl& c = a.ctl[t.slot];
  const int ev = c.ev;
  if (c.status != ST_RUNNING || ev == EV_NONE || ev == EV_ION || ev == EV_FORCE || ev == EV_STRESS) return;
  const int g = t.a, kx = t.b, half = t.c;
  if constexpr (KS == KS_WGC) {
    if (s.group_kind[g] == G_WGC3) {
      yz_wgc3_block<T>(a, s, g, kx, half, (cx<T>*)smem, tid, nthr);
      return;
    }
  }
  const int n2 = s.n2, n3 = s.zh, P = odd_pitch(n2);
  const size_t at = (size_t)kx * (n2 * s.n3) + half * n3 * n2;
  const int kind = s.group_kind[g];
  cx<T>* plane = (cx<T>*)s.spec + (size_t)s.group_f0[g] * (size_t)s.Nc + at;
  cx<T>* buf = (cx<T>*)smem;
  const StagePlan& py = s.qy;
  const StagePlan& pz = s.qzh;
  const unsigned mn2 = magic32(n2), mn3 = magic32(n3);
  const PlaneIO<T> glob{plane, n2}, rows{buf, P};
  ip_stage_acc<T, -1>(glob, rows, n2, mn2, pz, 0, a.tw, tid, nthr);
  BLOCK_SYNC();
  for (int st = 1; st < pz.nst; ++st) {
    ip_stage<T, -1>(buf, n2, mn2, 1, P, pz, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  for (int st = 0; st < py.nst - 1; ++st) {
    ip_stage<T, -1>(buf, n3, mn3, P, 1, py, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  if (kind == G_KMUL) {
    const KernOp<T> op{(const T*)s.kern + at, (T)s.inv_n, n2};
    ip_stage_op<T>(buf, n3, mn3, P, 1, py, op, tid, nthr);
  } else {
    GOp<T> op;
    op.gf.init(s);
    op.kind = kind;
    op.kx = kx;
    op.n2 = n2;
    op.n3 = s.n3;
    op.permy = a.idx + py.perm;
    op.permz = a.idx + s.qz.perm + half * n3;
    ip_stage_op<T>(buf, n3, mn3, P, 1, py, op, tid, nthr);
  }
  BLOCK_SYNC();
  for (int st = py.nst - 2; st >= 0; --st) {
    ip_stage<T, 1>(buf, n3, mn3, P, 1, py, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  for (int st = pz.nst - 1; st >= 1; --st) {
    ip_stage<T, 1>(buf, n2, mn2, 1, P, pz, st, a.tw, tid, nthr);
    BLOCK_SYNC();
  }
  ip_stage_acc<T, 1>(rows, glob, n2, mn2, pz, 0, a.tw, tid, nthr);
}

// ------------------------------------------------------------ pass 5
// Perdew-Zunger LDA potential and energy density (XC_LDA.f90:51-310) from
// rho, r13 = rho^(1/3), rs = cC / r13 and sr = sqrt(rs).
template <typename T>
HD void lda_point(T rho, T r13, T rs, T sr, T& vxc, T& exc) {
  const T cXp = T(-0.98474502184269641), cXe = T(-0.73855876638202234);
  if (rs < T(1)) {
    const T lr = m_log(rs);
    vxc = cXp * r13 + lr * (T(3.11e-2) + T(1.33333333333333333e-3) * rs) + T(-5.83666666666666666e-2) +
          T(-8.4e-3) * rs;
    exc = cXe * rho * r13 + rho * (lr * (T(3.11e-2) + T(2e-3) * rs) + T(-4.8e-2) + T(-1.16e-2) * rs);
  } else {
    const T den = T(1) + T(1.0529) * sr + T(3.334e-1) * rs;
    const T iden = T(1) / den;
    vxc = cXp * r13 + (T(-1.423e-1) + T(-0.174798948333333333) * sr + T(-6.325709333333333333e-2) * rs) *
                          (iden * iden);
    exc = cXe * rho * r13 + rho * (T(-1.423e-1) * iden);
  }
}

// All nf fields of a row-pair range are transformed as one batch of nf*nb
// sequences laid out [i][f*nb + b]; then every point of the rows gets the
// real-space epilogue.
// Inputs of the real-space epilogue of pass 5 (one task).
template <typename T>
struct XinvEpi {
  EvalIn<T> in;
  FieldPar<T> fp;
  const T* vion;
  T* w0;
  T* w1;
  T* trial;
  const T* bb;
  const cx<T>* res;  // the c2r outputs, column f*nc + col*nb + b, element i at res[i*es + column]
  int es, nb, nf, n1, u0;
  RowMap rm;
  bool opt_sqrt;
  T lam, muv, al, be, cTF, mu0, ieps, st, ctd, ctf53;
};

// The epilogue of one point: its potential (stored to the mode's output
// arrays at idx) and its terms of the mode's sums, added to sums[] in the
// slot precision.  o[f] are the point's field outputs of the inverse
// transforms; vi its ion potential, phin, rho, sq = sqrt(rho), y = rho^(-1/6)
// and x = rho^(-1/3) its evaluation input, ex and ey its optimiser inputs.
template <typename T, int EV>
HD void epi_input(const XinvEpi<T>& e, T aa, T bx, T& phin, T& rho, T& sq) {
  if (EV == EV_RHO) {  // the input is rho itself
    rho = aa;
    sq = m_sqrt(rho);
    phin = sq;
  } else {
    phin = phi_in(e.in.ca, aa, e.in.cb, bx);
    rho = phin * phin;
    sq = phin < T(0) ? -phin : phin;
  }
}
template <typename T, int KS, int EV, bool ENERGY>
HD void epi_point(const XinvEpi<T>& e, const T* o, T vi, T phin, T rho, T sq, T y, T x, T ex, T ey, int idx,
                  T* sums) {
  const FieldPar<T> fp = e.fp;
  const T cC = T(0.62035049089940009);
  const T r13 = sq * y;            // rho^(1/3)
  const T r23 = r13 * r13;
  const T rinv = x * x * x;        // 1/rho
  T vxc, exc;
  const T rs = cC * x;
  lda_point(rho, r13, rs, T(0.78762331789974329708) * y, vxc, exc);  // sqrt(cC) y
  T vnl, enl, lap;
  const T al = e.al, be = e.be, cTF = e.cTF;
  if constexpr (KS == KS_WT) {
    const T pa = e.nf > 3 ? o[3] : o[1];
    if (fp.pow56) {  // rho^(5/6) = rho y
      vnl = cTF * y * (al * o[1] + be * pa);
      enl = cTF * (rho * y) * o[1];
    } else {
      const T rbeta = m_pow(rho, be);
      const T ralpha = fp.aeqb ? rbeta : m_pow(rho, al);
      vnl = cTF * (al * (ralpha * rinv) * o[1] + be * (rbeta * rinv) * pa);
      enl = cTF * ralpha * o[1];
    }
    lap = o[2];
  } else {
    const T th = rho - fp.rho_s;
    const T ralpha = m_pow(rho, al);
    const T rbeta = fp.sum53 ? rho * r23 / ralpha : m_pow(rho, be);
    vnl = cTF * ((rbeta * rinv) * (be * o[2] + (rho + be * th) * o[3] + th * (rho + be * th * T(0.5)) * o[4]) +
                 (ralpha * rinv) * (al * o[5] + (rho + al * th) * o[6] + th * (rho + al * th * T(0.5)) * o[7]));
    enl = cTF * rbeta * (o[2] + th * o[3] + th * th * T(0.5) * o[4]);
    lap = o[1];
  }
  const T potr = vi + o[0] + vxc + e.ctf53 * r23 + vnl;
  const T muv = e.muv;
  const T pot = e.opt_sqrt ? T(2) * sq * potr + muv * lap : potr + muv * lap * (T(0.5) * sq * rinv);
  if constexpr (ENERGY) {
    sums[CH_EIE] += rho * vi;
    sums[CH_EH] += T(0.5) * o[0] * rho;
    sums[CH_EXC] += exc;
    sums[CH_ETF] += e.lam * cTF * (rho * r23);
    sums[CH_EVW] += T(0.5) * muv * sq * lap;
    sums[CH_ENL] += enl;
  }
  const T sg = phin < T(0) ? T(-1) : T(1);
  if constexpr (EV == EV_RHO) {
    e.w0[idx] = pot;
  } else if constexpr (EV == EV_PHI) {
    const T gg = pot * sg;
    e.w0[idx] = gg;
    sums[CH_M0] += gg * phin;
    sums[CH_M1] += phin * phin;
  } else if constexpr (EV == EV_CG) {
    const T gg = pot * sg;
    const T ap = ((gg - e.mu0 * T(2) * phin) - ex) * e.ieps;
    e.w1[idx] = ap;
    sums[CH_M0] += ey * ap;
  } else {  // EV_LS
    const T gg = pot * sg;
    e.w1[idx] = gg;
    e.trial[idx] = phin;
    const T dir = -ex * e.st + ey * e.ctd;
    const T dl = gg - T(2) * phin * e.mu0;
    sums[CH_M0] += gg * dir;
    sums[CH_M1] += dl * dl;
    sums[CH_M2] += gg * phin;
    sums[CH_M3] += phin * phin;
  }
}

// The epilogue over every point of the task, compiled per evaluation mode EV
// (ENERGY: the six energy channels are summed), so that each loop keeps only
// its own inputs and accumulators live.  A work item is one complex output
// of the inverse transforms: x index i of a column, whose real and imaginary
// parts are the points of its two rows (consecutive threads take consecutive
// i, so every global access is coalesced).  The two points'
// terms are added in the slot precision, then accumulated in FP64; the sums
// go to acc_out[NCH].
template <typename T, int KS, int EV, bool ENERGY>
HD void xinv_points(const XinvEpi<T>& e, double* acc_out, int tid, int nthr) {
  constexpr int NFM = KinFields<KS>::value;
  const T* __restrict__ vion = e.vion;
  const T* __restrict__ A = e.in.A;
  const T* __restrict__ B = e.in.B;
  const T* __restrict__ bb = e.bb;
  const int es = e.es, nb = e.nb, nf = e.nf, n1 = e.n1, zs = e.rm.zs, nc = zs * nb;
  double acc[NCH];
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) acc[ch] = 0.0;
  const unsigned mn1 = magic32(n1);
  for (int w = tid; w < nc * n1; w += nthr) {
    const int cb = magic_div32(w, mn1), i = w - cb * n1;
    const int col = cb >= nb ? 1 : 0, b = cb - col * nb;
    const bool has1 = e.rm.has1(e.u0 + b);
    const int idx0 = e.rm.row(e.u0 + b, col) * n1 + i, idx1 = has1 ? idx0 + n1 : idx0;
    // every global load of both points first
    const T vi0 = vion[idx0], vi1 = vion[idx1];
    const T aa0 = A[idx0], aa1 = A[idx1];
    // the second input (p in CG evaluations, d in line searches; the first
    // evaluation of a solve has none: its coefficient is 0)
    constexpr bool HASB = EV == EV_CG || EV == EV_LS;
    const T bx0 = HASB ? B[idx0] : T(0), bx1 = HASB ? B[idx1] : T(0);
    // the CG evaluation's second input is p, the line search's are phi and d
    const T ex0 = EV == EV_CG ? bb[idx0] : EV == EV_LS ? aa0 : T(0);
    const T ex1 = EV == EV_CG ? bb[idx1] : EV == EV_LS ? aa1 : T(0);
    T o0[NFM], o1[NFM];
    const cx<T>* rv = e.res + i * es + cb;
#pragma unroll
    for (int f = 0; f < NFM; ++f) {
      const cx<T> z = f < nf ? rv[f * nc] : mk<T>(T(0), T(0));
      o0[f] = z.x;
      o1[f] = z.y;
    }
    T sums[NCH];
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) sums[ch] = T(0);
    T p0, p1, rho0, rho1, sq0, sq1;
    epi_input<T, EV>(e, aa0, bx0, p0, rho0, sq0);
    epi_input<T, EV>(e, aa1, bx1, p1, rho1, sq1);
    T y0, y1, x0, x1;
    m_icbrt2(sq0, y0, x0);
    m_icbrt2(sq1, y1, x1);
    if (icbrt_out(sq0) || icbrt_out(sq1)) {
      y0 = m_icbrt_any(sq0);
      y1 = m_icbrt_any(sq1);
      x0 = m_icbrt_any(rho0);
      x1 = m_icbrt_any(rho1);
    }
    epi_point<T, KS, EV, ENERGY>(e, o0, vi0, p0, rho0, sq0, y0, x0, ex0, bx0, idx0, sums);
    if (has1) epi_point<T, KS, EV, ENERGY>(e, o1, vi1, p1, rho1, sq1, y1, x1, ex1, bx1, idx1, sums);
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) acc[ch] += (double)sums[ch];
  }
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) acc_out[ch] = acc[ch];
}

template <typename T, int KS>
HD void xinv_block(const Args<T>& a, int bid, int tid, int nthr, char* smem) {
  const Task t = a.tasks[bid];
  SlotDev& s = a.slots[t.slot];
  Ctl& c = a.ctl[t.slot];
  const int ev = c.ev;
  if (c.status != ST_RUNNING || ev == EV_NONE) return;
  const int u0 = t.a, nb = t.b, ordinal = t.c;
  const bool setup_mode = ev == EV_ION || ev == EV_FORCE;
  const int n1 = s.n1;
  const int nf = ev == EV_ION ? 1 : ev == EV_FORCE ? s.ion.nspec : s.nf;
  const int nc = s.zs * nb, NB = nf * nc;
  const long long Nc = s.Nc;
  const cx<T>* __restrict__ spec = (const cx<T>*)s.spec;
  cx<T>* buf = (cx<T>*)smem;
  double* sred = (double*)(smem + xinv_buf(n1, nf, nc, sizeof(T)));
  if (ev == EV_STRESS) {  // the spectra stay; no sums
    double zero[NCH];
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) zero[ch] = 0.0;
    store_partials<0, 0>(s, ordinal, zero, sred, tid, nthr);
    return;
  }
  const int es = x_pitch(NB);
  const RowMap rm = row_map(s);
  x_gather<T>(buf, spec, Nc, rm, u0, nf, nb, es, s.qx, a.idx + s.qx.iperm, a.tw + s.qz.root, tid, nthr);
  BLOCK_SYNC();
  {
    const unsigned mcols = magic32(NB);
    for (int st = s.qx.nst - 1; st >= 0; --st) {
      ip_stage<T, 1>(buf, NB, mcols, 1, es, s.qx, st, a.tw, tid, nthr);
      BLOCK_SYNC();
    }
  }
  const cx<T>* res = buf;
  if (setup_mode) {
    // EV_ION: ionPotReal; EV_FORCE: the per-species Factor arrays in buf[B_B + s]
    const unsigned mn1s = magic32(n1);
    for (int w = tid; w < nc * n1; w += nthr) {
      const int cb = magic_div32(w, mn1s), i = w - cb * n1;
      const int col = cb >= nb ? 1 : 0, b = cb - col * nb;
      const int i0 = rm.row(u0 + b, col) * n1 + i;
      for (int f = 0; f < nf; ++f) {
        const cx<T> z = res[i * es + f * nc + cb];
        T* dst = ev == EV_ION ? (T*)s.vion : (T*)s.buf[B_B + f];
        dst[i0] = z.x;
        if (rm.has1(u0 + b)) dst[i0 + n1] = z.y;
      }
    }
    double zero[NCH];
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) zero[ch] = 0.0;
    store_partials<0, 0>(s, ordinal, zero, sred, tid, nthr);
    return;
  }

  XinvEpi<T> e;
  e.in = eval_in<T>(s, c);
  e.fp = field_par<T>(s);
  e.vion = (const T*)s.vion;
  e.w0 = (T*)s.buf[c.iw0];
  e.w1 = (T*)s.buf[c.iw1];
  e.trial = (T*)s.buf[c.itrial];
  e.bb = (const T*)s.buf[B_B];
  e.res = res;
  e.es = es;
  e.nb = nb;
  e.nf = nf;
  e.n1 = n1;
  e.rm = rm;
  e.u0 = u0;
  e.opt_sqrt = c.opt_sqrt != 0 || ev != EV_RHO;
  e.lam = (T)s.lambda;
  e.muv = (T)s.mu;
  e.al = e.fp.alpha;
  e.be = e.fp.beta;
  e.cTF = (T)C_TF;
  e.mu0 = (T)c.mu;
  e.ieps = (T)(ev == EV_CG ? 1.0 / c.eps : 0.0);
  e.st = (T)c.st;
  e.ctd = (T)(c.ct * c.dscale);
  e.ctf53 = T(5) / T(3) * e.cTF * e.lam;
  double acc[NCH];
  switch (ev) {
    case EV_CG:
      xinv_points<T, KS, EV_CG, false>(e, acc, tid, nthr);
      break;
    case EV_LS:
      xinv_points<T, KS, EV_LS, true>(e, acc, tid, nthr);
      break;
    case EV_PHI:
      xinv_points<T, KS, EV_PHI, true>(e, acc, tid, nthr);
      break;
    default:
      if (c.want_energy) xinv_points<T, KS, EV_RHO, true>(e, acc, tid, nthr);
      else xinv_points<T, KS, EV_RHO, false>(e, acc, tid, nthr);
      break;
  }
  if (ev == EV_CG) store_partials<CH_M0, CH_M0 + 1>(s, ordinal, acc, sred, tid, nthr);
  else store_partials(s, ordinal, acc, sred, tid, nthr);
}

}  // namespace ofdft
