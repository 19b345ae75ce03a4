// What the FP64 passes (passes.cuh) and the FP32 passes (f32/passes.cuh) share:
// the kernels' arguments, the ion potential's spline, block reductions, the
// controller and vector kernels' bodies, the evaluation's inputs and the
// k-space factors.
#pragma once
#include "ntn_ctl.cuh"

namespace ofdft {

constexpr double PI_D = 3.141592653589793238462643;
constexpr double C_TF = 2.87123400018819;  // Source/KEDF_TF.f90:42

// Kernel instantiations per kinetic functional: the WT kernels carry at most
// 4 fields and no WGC code, so their register allocation is not set by the
// 8-field WGC paths.
enum KinSel : int { KS_WT = 0, KS_WGC = 1 };
template <int KS> struct KinFields { static constexpr int value = KS == KS_WT ? 4 : MAX_FIELDS; };

template <typename T>
struct Args {
  SlotDev* slots;
  Ctl* ctl;
  const Task* tasks;
  const cx<T>* tw;   // roots of unity of every length (FftPlan::root); FP64: and stage twiddles (StagePlan::stw)
  const int* idx;    // digit-reversal tables (FftPlan::perm, iperm)
  int vchunk;        // points per task of the vector kernel
};

HD size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// V_loc(|q|) by the index-knot cubic spline (PspRecipCubicSpline, LocalPseudoPot.f90:92-202).
HD double psp_value(const IonAux& x, int sp, double q) {
  const PspDev& p = x.psp[sp];
  if (q == 0.0) return p.v0;
  if (q >= p.max_g) return 0.0;
  const double pos = q / p.dq + 1.0;
  const int left = (int)floor(pos);
  const double dt = pos - (double)left;
  const double* vqs = x.tab + p.off;
  const double* pdd = x.tab + p.off + p.npts;
  const double yl = vqs[left - 1], yr = vqs[left];
  const double pl = pdd[left - 1], pr = pdd[left];
  const double yval = yl + dt * (yr - yl - (pr / 6.0 + pl / 3.0) + dt * (0.5 * pl + dt * ((pr - pl) / 6.0)));
  return yval - 4.0 * PI_D * p.charge / (q * q);
}

// ------------------------------------------------------------ reductions
// Reduce channels [LO, HI) of acc[NCH] over the block; the block totals end
// up in sred[LO..HI-1] and the other channels of sred[0..NCH-1] are zero.  On
// the device: warp shuffles, then one warp over the per-warp sums (sred needs
// NCH * 33 doubles).  In the host emulation the block has one thread.  Passes
// whose sums use few channels (a CG evaluation one, the vector operations
// three) reduce only those.
template <int LO = 0, int HI = NCH>
HDNI inline void block_reduce(double* sred, const double* acc, int tid, int nthr) {
#if defined(__CUDA_ARCH__)
  const int lane = tid & 31, warp = tid >> 5, nw = (nthr + 31) >> 5;
  double v[NCH];
#pragma unroll
  for (int ch = LO; ch < HI; ++ch) {
    double x = acc[ch];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    v[ch] = x;
  }
  if (lane == 0) {
#pragma unroll
    for (int ch = LO; ch < HI; ++ch) sred[NCH + ch * 32 + warp] = v[ch];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      if (ch < LO || ch >= HI) {
        if (lane == 0) sred[ch] = 0.0;
        continue;
      }
      double x = lane < nw ? sred[NCH + ch * 32 + lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) sred[ch] = x;
    }
  }
  __syncthreads();
#else
  (void)tid;
  (void)nthr;
  for (int ch = 0; ch < NCH; ++ch) sred[ch] = (ch >= LO && ch < HI) ? acc[ch] : 0.0;
#endif
}

// Store this task's per-channel sums (channels [LO, HI), the rest zero) in
// the slot's partials.
template <int LO = 0, int HI = NCH>
HDNI inline void store_partials(SlotDev& s, int task_idx, const double* acc, double* sred, int tid, int nthr) {
  block_reduce<LO, HI>(sred, acc, tid, nthr);
  if (tid == 0) {
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) s.partials[(size_t)task_idx * NCH + ch] = sred[ch];
  }
}

// Shared memory of the controller block: the reduction scratch, then a copy
// of the slot's controller record.
constexpr size_t CTL_SRED_BYTES = (NCH * 33 + 2) * sizeof(double);
constexpr size_t CTL_SMEM_BYTES = CTL_SRED_BYTES + sizeof(Ctl);
static_assert(sizeof(Ctl) % 8 == 0, "the controller record is copied as 8-byte words");

// Copy nbytes (a multiple of 8) as 8-byte words spread over the block.
HDNI inline void copy_words(void* dst, const void* src, size_t nbytes, int tid, int nthr) {
  unsigned long long* d = (unsigned long long*)dst;
  const unsigned long long* s = (const unsigned long long*)src;
  for (int w = tid; w < (int)(nbytes / 8); w += nthr) d[w] = s[w];
}

// Controller kernel body, one block per running slot: reduce the partials
// of the work kernel that just ran (in a fixed order, independent of block
// scheduling) and advance the slot's NTN state machine.  kid = K_VEC after the
// vector kernel, K_X5 after pass 5.  The block copies the controller record
// into shared memory with all its threads; the one thread that runs the
// state machine reads and writes only the fields it needs there, and the
// block writes the record back.
HDNI inline void ctl_block(SlotDev* slots, Ctl* ctls, const Task* tasks, int kid, int bid, int tid, int nthr,
                           char* smem) {
  const int si = tasks[bid].slot;
  SlotDev& s = slots[si];
  Ctl& c = ctls[si];
  if (c.status != ST_RUNNING) return;
  const int what = kid == K_VEC ? c.op : c.ev;
  if (what == 0) return;
  double* sred = (double*)smem;
  Ctl* cs = (Ctl*)(smem + CTL_SRED_BYTES);
  copy_words(cs, &c, sizeof(Ctl), tid, nthr);
  const CtlSlot sl = ctl_slot(s);
  const int nt = s.ntask[kid];
  double part[NCH];
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) part[ch] = 0.0;
  for (int t = tid; t < nt; t += nthr) {
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) part[ch] += s.partials[(size_t)t * NCH + ch];
  }
  block_reduce(sred, part, tid, nthr);  // its barriers also publish the copy
  if (tid == 0) {
    double red[NCH];
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) red[ch] = sred[ch];
    ntn_after(*cs, sl, red, kid, what);
  }
  BLOCK_SYNC();
  copy_words(&c, cs, sizeof(Ctl), tid, nthr);
}

// ------------------------------------------------------------ vector ops
// 16-byte packs (4 floats or 2 doubles): the vector operations stream their
// arrays with one 16-byte load or store per pack and array.
template <typename T> struct Pack { static constexpr int n = 16 / (int)sizeof(T); };
template <typename T>
HD void ld_pack(T* v, const T* p) {
#if defined(__CUDA_ARCH__)
  if constexpr (sizeof(T) == 4) {
    const float4 x = *(const float4*)p;
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  } else {
    const double2 x = *(const double2*)p;
    v[0] = x.x; v[1] = x.y;
  }
#else
  for (int l = 0; l < Pack<T>::n; ++l) v[l] = p[l];
#endif
}
template <typename T>
HD void st_pack(T* p, const T* v) {
#if defined(__CUDA_ARCH__)
  if constexpr (sizeof(T) == 4) *(float4*)p = make_float4(v[0], v[1], v[2], v[3]);
  else *(double2*)p = make_double2(v[0], v[1]);
#else
  for (int l = 0; l < Pack<T>::n; ++l) p[l] = v[l];
#endif
}

// One task of a vector operation over points [i0, i1) of a slot: packs of
// Pack<T>::n points first (i0 is a multiple of the chunk size, so packs are
// 16-byte aligned), then the points after the last full pack one at a time.
template <typename T>
HD void vec_block(const Args<T>& a, int bid, int tid, int nthr, char* smem) {
  const Task t = a.tasks[bid];
  SlotDev& s = a.slots[t.slot];
  Ctl& c = a.ctl[t.slot];
  const int op = c.op;
  if (c.status != ST_RUNNING || op == OP_NONE) return;
  T* __restrict__ phi = (T*)s.buf[c.iphi];
  const T* __restrict__ w0 = (const T*)s.buf[c.iw0];
  const T* __restrict__ w1 = (const T*)s.buf[c.iw1];
  T* __restrict__ bb = (T*)s.buf[B_B];
  T* __restrict__ r = (T*)s.buf[B_R];
  T* __restrict__ p = (T*)s.buf[B_P];
  T* __restrict__ d = (T*)s.buf[B_D];
  const T k = (T)c.opc;
  const int i0 = t.a * a.vchunk;
  const int n = (int)s.N;
  const int i1 = i0 + a.vchunk < n ? i0 + a.vchunk : n;
  constexpr int VP = Pack<T>::n;
  const int npk = (i1 - i0) / VP;  // full packs
  const int it = i0 + npk * VP;    // first point after them
  double acc[NCH];
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) acc[ch] = 0.0;
  switch (op) {
    case OP_SQRT_INIT:
      for (int q = tid; q < npk; q += nthr) {
        const int i = i0 + q * VP;
        T v[VP];
        ld_pack(v, phi + i);
#pragma unroll
        for (int l = 0; l < VP; ++l) {
          acc[0] += (double)v[l];
          v[l] = m_sqrt(v[l] < T(0) ? -v[l] : v[l]);
        }
        st_pack(phi + i, v);
      }
      for (int i = it + tid; i < i1; i += nthr) {
        const T rho = phi[i];
        acc[0] += (double)rho;
        phi[i] = m_sqrt(rho < T(0) ? -rho : rho);
      }
      break;
    case OP_DLDPHI:
      for (int q = tid; q < npk; q += nthr) {
        const int i = i0 + q * VP;
        T wv[VP], fv[VP], bv[VP], rv[VP], zv[VP];
        ld_pack(wv, w0 + i);
        ld_pack(fv, phi + i);
#pragma unroll
        for (int l = 0; l < VP; ++l) {
          const T v = wv[l] - k * T(2) * fv[l];
          bv[l] = v;
          rv[l] = -v;
          zv[l] = T(0);
          acc[0] += (double)v * (double)v;
        }
        st_pack(bb + i, bv);
        st_pack(r + i, rv);
        st_pack(p + i, rv);
        st_pack(d + i, zv);
      }
      for (int i = it + tid; i < i1; i += nthr) {
        const T v = w0[i] - k * T(2) * phi[i];
        bb[i] = v;
        r[i] = -v;
        p[i] = -v;
        d[i] = T(0);
        acc[0] += (double)v * (double)v;
      }
      break;
    case OP_CGSTEP:
      for (int q = tid; q < npk; q += nthr) {
        const int i = i0 + q * VP;
        T dv[VP], pv[VP], rv[VP], wv[VP], fv[VP];
        ld_pack(dv, d + i);
        ld_pack(pv, p + i);
        ld_pack(rv, r + i);
        ld_pack(wv, w1 + i);
        ld_pack(fv, phi + i);
#pragma unroll
        for (int l = 0; l < VP; ++l) {
          const T dn = dv[l] + k * pv[l];
          const T rn = rv[l] - k * wv[l];
          dv[l] = dn;
          rv[l] = rn;
          const T pd = fv[l] + dn;
          acc[0] += (double)rn * (double)rn;
          acc[1] += (double)pd * (double)pd;
          acc[2] += (double)fv[l] * (double)dn;
        }
        st_pack(d + i, dv);
        st_pack(r + i, rv);
      }
      for (int i = it + tid; i < i1; i += nthr) {
        const T dn = d[i] + k * p[i];
        const T rn = r[i] - k * w1[i];
        d[i] = dn;
        r[i] = rn;
        const T f = phi[i];
        const T pd = f + dn;
        acc[0] += (double)rn * (double)rn;
        acc[1] += (double)pd * (double)pd;
        acc[2] += (double)f * (double)dn;
      }
      break;
    case OP_PUPD:
      for (int q = tid; q < npk; q += nthr) {
        const int i = i0 + q * VP;
        T rv[VP], pv[VP];
        ld_pack(rv, r + i);
        ld_pack(pv, p + i);
#pragma unroll
        for (int l = 0; l < VP; ++l) {
          pv[l] = rv[l] + k * pv[l];
          acc[0] += (double)pv[l] * (double)pv[l];
        }
        st_pack(p + i, pv);
      }
      for (int i = it + tid; i < i1; i += nthr) {
        const T pn = r[i] + k * p[i];
        p[i] = pn;
        acc[0] += (double)pn * (double)pn;
      }
      break;
    case OP_DIRNEG:
    case OP_NG1:
    case OP_SD:
      for (int q = tid; q < npk; q += nthr) {
        const int i = i0 + q * VP;
        T dv[VP], fv[VP], xv[VP];
        if (op == OP_DIRNEG) {
          ld_pack(dv, d + i);
          ld_pack(xv, p + i);
        } else if (op == OP_SD) {
          ld_pack(xv, bb + i);
        } else {
          ld_pack(dv, d + i);
        }
        ld_pack(fv, phi + i);
#pragma unroll
        for (int l = 0; l < VP; ++l) {
          T dn;
          if (op == OP_DIRNEG) dn = -(dv[l] - k * xv[l]);
          else if (op == OP_SD) dn = -xv[l];
          else dn = dv[l];
          dv[l] = dn;
          const T pd = fv[l] + dn;
          acc[1] += (double)pd * (double)pd;
          acc[2] += (double)fv[l] * (double)dn;
        }
        if (op != OP_NG1) st_pack(d + i, dv);
      }
      for (int i = it + tid; i < i1; i += nthr) {
        T dn;
        if (op == OP_DIRNEG) dn = -(d[i] - k * p[i]);
        else if (op == OP_SD) dn = -bb[i];
        else dn = d[i];
        if (op != OP_NG1) d[i] = dn;
        const T f = phi[i];
        const T pd = f + dn;
        acc[1] += (double)pd * (double)pd;
        acc[2] += (double)f * (double)dn;
      }
      break;
    case OP_NG2:
      for (int q = tid; q < npk; q += nthr) {
        const int i = i0 + q * VP;
        T dv[VP], fv[VP], wv[VP];
        ld_pack(dv, d + i);
        ld_pack(fv, phi + i);
        ld_pack(wv, w0 + i);
#pragma unroll
        for (int l = 0; l < VP; ++l) {
          const T dn = dv[l] - fv[l] * k;
          dv[l] = dn;
          acc[0] += (double)dn * (double)dn;
          acc[1] += (double)wv[l] * (double)dn;
        }
        st_pack(d + i, dv);
      }
      for (int i = it + tid; i < i1; i += nthr) {
        const T dn = d[i] - phi[i] * k;
        d[i] = dn;
        acc[0] += (double)dn * (double)dn;
        acc[1] += (double)w0[i] * (double)dn;
      }
      break;
    default:
      break;
  }
  store_partials<0, 3>(s, t.a, acc, (double*)smem, tid, nthr);  // vector ops use channels 0-2
}

// ------------------------------------------------------------ evaluation inputs
// phi_in = ca * A + cb * B of the current evaluation (or rho itself for the
// drop-in evaluation), held in registers for a whole block.
template <typename T>
struct EvalIn {
  const T* __restrict__ A;
  const T* __restrict__ B;
  T ca, cb;
  int rho_mode;
};

template <typename T>
HD EvalIn<T> eval_in(const SlotDev& s, const Ctl& c) {
  EvalIn<T> e;
  e.A = (const T*)s.buf[c.iphi];
  e.B = (const T*)s.buf[c.evb];
  e.ca = (T)c.ca;
  e.cb = (T)c.cb;
  e.rho_mode = (c.ev == EV_RHO || c.ev == EV_STRESS || (c.ev == EV_FORCE && c.force_rho)) ? 1 : 0;
  return e;
}

// Functional parameters of the real-space stages, in registers.
template <typename T>
struct FieldPar {
  int wt, pow56, aeqb, sum53;
  T alpha, beta, rho_s;
};

template <typename T>
HD FieldPar<T> field_par(const SlotDev& s) {
  FieldPar<T> f;
  f.wt = s.kinetic == KIN_WT;
  f.pow56 = s.pow56;
  f.aeqb = s.alpha_eq_beta;
  f.sum53 = (s.alpha + s.beta - 5.0 / 3.0) < 1e-14 && (s.alpha + s.beta - 5.0 / 3.0) > -1e-14;
  f.alpha = (T)s.alpha;
  f.beta = (T)s.beta;
  f.rho_s = (T)s.rho_s;
  return f;
}

// ------------------------------------------------------------ k-space operators
HD int signed_freq(int k, int n) { return k > n / 2 ? k - n : k; }

// Real factor of the single-field operators at the frequency (m1, m2, m3)
// (signed): Hartree 4 pi / |G|^2 (0 at G = 0) and vW |G|^2, each times the
// 1/N forward scale; |G|^2 in the slot's precision.
template <typename T>
struct GFactor {
  T rt[9];
  T sc, c4;
  HD void init(const SlotDev& s) {
#pragma unroll
    for (int q = 0; q < 9; ++q) rt[q] = (T)s.recip[q];
    sc = (T)s.inv_n;
    c4 = (T)(4.0 * PI_D * s.inv_n);
  }
  HD T operator()(int kind, int m1, int m2, int m3) const {
    const T tx = rt[0] * (T)m1 + rt[3] * (T)m2 + rt[6] * (T)m3;
    const T ty = rt[1] * (T)m1 + rt[4] * (T)m2 + rt[7] * (T)m3;
    const T tz = rt[2] * (T)m1 + rt[5] * (T)m2 + rt[8] * (T)m3;
    const T g2 = tx * tx + ty * ty + tz * tz;
    if (kind == G_VW) return g2 * sc;
    return (m1 == 0 && m2 == 0 && m3 == 0) ? T(0) : c4 / g2;
  }
};

// Odd row pitch of a plane or tile held in shared memory with y fastest:
// transforms along y then take columns at an odd stride (conflict-free).
HD int odd_pitch(int n) { return n | 1; }

// Accessors of the fused pass: the plane in global memory (y fastest, row
// length n2) and in shared memory (rows of odd pitch P); column c is y,
// position i is z.
template <typename T>
struct PlaneIO {
  cx<T>* p;
  int pitch;
  HD cx<T> ld(int y, int z) const { return p[z * pitch + y]; }
  HD void st(int y, int z, cx<T> v) const { p[z * pitch + y] = v; }
};

// Operator factor at (column z, y position q) of the fused pass: the WT kernel
// plane (stored in the transforms' digit-reversed order) times the 1/N forward
// scale.
template <typename T>
struct KernOp {
  const T* __restrict__ kern;
  T sc;
  int n2;
  HD T operator()(int z, int q) const { return kern[z * n2 + q] * sc; }
};

// The (y, z) planes at kx of the three fields of a WGC group in the spectra
// (field p at base + p*Nc), seen as 3*n2 columns c = p*n2 + y of n3
// positions z.
template <typename T>
struct Planes3IO {
  cx<T>* base;
  long long Nc;
  int n2;
  unsigned mn2;
  HD size_t at(int c, int z) const {
    const int p = magic_div32(c, mn2), y = c - p * n2;
    return (size_t)p * (size_t)Nc + (size_t)z * n2 + y;
  }
  HD cx<T> ld(int c, int z) const { return base[at(c, z)]; }
  HD void st(int c, int z, cx<T> v) const { base[at(c, z)] = v; }
};

}  // namespace ofdft
