// Stress tensor of a density on the device (CalculateStress,
// Source/CalStress.f90:44-253) for the WT and second-order WGC functionals
// with LDA exchange-correlation, the B-spline ion-electron term and the
// Ewald sum.
//
// The density's forward spectra (rho, rho^beta, sqrt(rho), rho^alpha) come
// from the engine's own transforms (EV_STRESS passes: x, y and z forward, in
// the kx-major, digit-reversed layout of the slot's spectra).  One reduction
// kernel then visits every stored frequency once and adds, in FP64,
//   vW        <d_a sqrt(rho) d_b sqrt(rho)> by Parseval over the full
//             spectrum (weight 2 off the kx = 0 and x-Nyquist planes; on
//             those planes, whose imaginary parts the c2r transform drops,
//             the derivative of a Nyquist index is that of index 0)
//                                                  (VWStress, KEDF_VW.f90:365-449)
//   WT        -eta G'(eta) Re(F[rho^a] F[rho^b]*) (q_a q_b / q^2, and its trace)
//                                                  (WTStress, KEDF_WT.f90:263-394)
//   WGC       the kernel-derivative sums of F[rho^x], x = a, b, a+1, b+1, a+2,
//             b+2 (stress_wgc_point)               (WGCStress, KEDF_WGC.f90:519-745)
//   Hartree   |rho(q)|^2 q_a q_b / q^4                (JStress, Hartree.f90:173-247)
//   ion-elec. Re(rho(q) S_s(q)) V_s'(q) q_a q_b / q, S_s the B-spline
//             structure factor of species s       (IonElectronStressSpline,
//                                                   IonElectronSpline.f90:359-534)
// over the half spectrum of qMask (PlaneWave.f90:255-296) for all but vW.
// The structure factor is the DFT of FillQIonTable's spread charges, taken
// ion by ion as a product of three 1D sums of the stencil weights
// (A_d(ion, k) = sum_i M_d[i] exp(-2 pi i k (i - floor_d) / n_d)), so no
// charge grid is built.  The Ewald stress adds the strain derivatives of the
// real- and reciprocal-space sums of ewald.cuh (EwaldStress,
// Ewald.f90:1857-2535) with the same splitting.  Sums run in a fixed order
// (per-thread, a fixed tree per block, blocks in index order on the host), so
// results do not depend on scheduling.
#pragma once

#include "cx.cuh"
#include "ewald.cuh"
#include "setup.cuh"

namespace ofdft {

// Accumulator channels of the spectral reduction: six upper-triangle
// components (xx, xy, xz, yy, yz, zz) per tensor term.
enum StressChannel : int { SC_VW = 0, SC_WT = 6, SC_WTTR = 12, SC_H = 13, SC_IE = 19, NSC = 25 };

struct StressArgs {
  const int* permy;          // digit-reversed position -> natural ky
  const int* permz;          // -> natural kz
  const cx<double>* sf;      // A_d(ion, k): per ion k1 + n2 + n3 entries (x, then y, then z)
  const int* species;        // species of each ion
  int nion;
  double kf;                 // (3 pi^2 rho0)^(1/3) (WT), (3 pi^2 rho*)^(1/3) (WGC)
  double ki, gamma;          // WGC: 20 rho0^(5/3 - alpha - beta), the kernel's gamma
};

// qMask (PlaneWave.f90:255-296) at natural indices (kx < k1, ky, kz): the
// half of the r2c spectrum without the conjugate partners on the kx = 0 and
// x-Nyquist planes and without their self-conjugate points.
HD bool stress_mask(int kx, int ky, int kz, int n1, int n2, int n3) {
  const bool h2 = ky >= 1 && ky <= (n2 - 1) / 2;
  const bool h3 = kz >= 1 && kz <= (n3 - 1) / 2;
  const bool plane = h2 || (ky == 0 && h3) || ((n2 % 2) == 0 && ky == n2 / 2 && h3);
  if (n1 % 2 == 1) {
    if (kx >= 1) return true;
  } else if (kx >= 1 && kx < n1 / 2) {
    return true;
  }
  if (kx == 0) return plane;
  return (n1 % 2) == 0 && kx == n1 / 2 && plane;
}

// dLindG/deta (GPrime, MathFunctions.f90:531-578) with the vW coefficient mu.
HD double wt_g_prime(double e, double mu) {
  if (e < 0.0) return 0.0;
  if (e < 1e-10) return 2.0 * e * (1.0 / 3.0 - 3.0 * mu);
  if (dabs(e - 1.0) < 1e-10) return 40.0;
  const double l1 = log(dabs((1.0 + e) / (1.0 - e)));
  const double l2 = log((1.0 + e) / dabs(1.0 - e));
  const double den = 0.5 + 0.25 * (1.0 - e * e) * l2 / e;
  return ((e * e + 1.0) * 0.25 / (e * e) * l1 - 0.5 / e) / (den * den) - 6.0 * e * mu;
}

// dV_loc/dq by the same index-knot spline as psp_value (PseudoPotDiffLookup,
// LocalPseudoPot.f90:207-276), plus the derivative of the -4 pi Z / q^2 tail.
HD double psp_diff(const IonAux& x, int sp, double q) {
  const PspDev& p = x.psp[sp];
  if (!(q > 0.0) || q > p.max_g) return 0.0;
  const double pos = q / p.dq + 1.0;
  int left = (int)floor(pos);
  if (left < 1) left = 1;
  if (left > p.npts - 1) left = p.npts - 1;
  const double dt = pos - (double)left;
  const double* vqs = x.tab + p.off;
  const double* pdd = x.tab + p.off + p.npts;
  const double yl = vqs[left - 1], yr = vqs[left];
  const double pl = pdd[left - 1], pr = pdd[left];
  const double yp = (yr - yl) - (pr / 6.0 + pl / 3.0) + dt * (pl + dt * 0.5 * (pr - pl));
  return yp / p.dq + 8.0 * PI_D * p.charge / (q * q * q);
}

// sin and cos of 2 pi t / n (0 <= t < n).
HD void sincos_turn(long long t, int n, double* sn, double* cs) {
#if defined(__CUDA_ARCH__)
  sincospi(2.0 * (double)t / (double)n, sn, cs);
#else
  const double a = 2.0 * PI_D * (double)t / (double)n;
  *sn = std::sin(a);
  *cs = std::cos(a);
#endif
}

// Entry w of ion i's table: A_d(i, k) for axis d (w < k1: x; then n2 y
// entries; then n3 z entries).  The phase k (j - floor) is reduced modulo
// n_d in integers first.
HD cx<double> stress_sf_entry(const SlotDev& s, const IonStencil& st, int w) {
  int d = 0, k = w, n = s.n1;
  if (w >= s.k1 + s.n2) {
    d = 2;
    k = w - s.k1 - s.n2;
    n = s.n3;
  } else if (w >= s.k1) {
    d = 1;
    k = w - s.k1;
    n = s.n2;
  }
  double re = 0.0, im = 0.0;
  for (int j = 0; j < SPLINE_ORDER; ++j) {
    long long t = ((long long)k * (long long)(j - st.fl[d])) % n;
    if (t < 0) t += n;
    double sn, cs;
    sincos_turn(t, n, &sn, &cs);
    re += st.M[d][j] * cs;
    im -= st.M[d][j] * sn;
  }
  return mk<double>(re, im);
}

template <typename T>
HD cx<double> spec_at(const SlotDev& s, int f, long long p) {
  const cx<T> v = ((const cx<T>*)s.spec)[(size_t)f * (size_t)s.Nc + (size_t)p];
  return mk<double>((double)v.x * s.inv_n, (double)v.y * s.inv_n);
}

// Re(conj(a) b).
HD double re_cb(cx<double> a, cx<double> b) { return a.x * b.x + a.y * b.y; }

// The WGC kinetic terms of one masked frequency (WGCStress, KEDF_WGC.f90:
// 519-745, WGCT = 2, rho0 and rho* refreshed with the cell): acc[SC_WTTR]
// gets the diagonal sum (diago + offdia diff), acc[SC_WT..] offdia q_a q_b / q^2;
// both are scaled by 2 cTF on the host.  F[rho^(x+1)] and F[rho^(x+2)] come
// from the evaluation's fields rho^x, theta rho^x, theta^2 rho^x / 2 (theta =
// rho - rho*) by linearity.
template <typename T>
HD void stress_wgc_point(const SlotDev& s, const StressArgs& sa, long long p, const double* g, double q2,
                         double eta, double* acc) {
  const double a = s.alpha, b = s.beta, rs = s.rho_s, gm = sa.gamma;
  const cx<double> A = spec_at<T>(s, 2, p), At = spec_at<T>(s, 3, p), Ah = spec_at<T>(s, 4, p);
  const cx<double> B = spec_at<T>(s, 5, p), Bt = spec_at<T>(s, 6, p), Bh = spec_at<T>(s, 7, p);
  const cx<double> A1 = mk<double>(At.x + rs * A.x, At.y + rs * A.y);
  const cx<double> B1 = mk<double>(Bt.x + rs * B.x, Bt.y + rs * B.y);
  const cx<double> A2 = mk<double>(2.0 * Ah.x + 2.0 * rs * At.x + rs * rs * A.x, 2.0 * Ah.y + 2.0 * rs * At.y + rs * rs * A.y);
  const cx<double> B2 = mk<double>(2.0 * Bh.x + 2.0 * rs * Bt.x + rs * rs * B.x, 2.0 * Bh.y + 2.0 * rs * Bt.y + rs * rs * B.y);
  const T* kern = (const T*)s.kern;
  const double K1 = (double)kern[p], K2 = (double)kern[s.Nc + p], K3 = (double)kern[2 * s.Nc + p],
               K4 = (double)kern[3 * s.Nc + p];
  // hold0 = holdS = .FALSE.
  const double c001 = -2.0 / 3.0, c002 = rs * 4.0 / 3.0, c003 = -rs * rs * 2.0 / 3.0;
  const double c011 = -5.0 / 3.0 + 1.0, c012 = rs * 5.0 / 3.0 - rs, c021 = -4.0 / 3.0 + 1.0, c111 = -8.0 / 3.0 + 2.0;
  const double diff = -1.0 / 3.0;
  const double c00 = c001 * K1 + c002 * K2 + c003 * (K3 + K4);
  const double c01 = c011 * K2 + c012 * (K3 + K4);
  const double c02 = c021 * K3;
  const double c11 = c111 * K4;
  const double p00 = re_cb(A, B), p10 = re_cb(A1, B), p01 = re_cb(A, B1), p20 = re_cb(A2, B), p02 = re_cb(A, B2),
               p11 = re_cb(A1, B1);
  const double diago = c00 * p00 + c01 * (p10 + p01) + c02 * (p20 + p02) + c11 * p11;
  const double gp = wt_g_prime(eta, s.mu);
  const double d11 = -sa.ki * eta / (36.0 * rs * rs) * gp - K4 * 6.0 * (a + b) - K2 * (gm * (a + b) + 6.0 * a * b) / rs;
  const double d02 = -sa.ki * eta / (72.0 * rs * rs) * gp - K4 * (3.0 * (a + b + 1.0) - gm) -
                     K2 * (3.0 * gm * (a + b + 1.0) - gm * gm + 18.0 * a * b) / (6.0 * rs);
  double d01 = K4 * 6.0 * rs + K2 * gm;
  const double d00 = 6.0 * rs * K2 - 2.0 * rs * d01 + rs * rs * (2.0 * d02 + d11);
  d01 = -rs * (d11 + 2.0 * d02) + d01;
  const double offdia = d00 * p00 + d01 * (p10 + p01) + d02 * (p20 + p02) + d11 * p11;
  acc[SC_WTTR] += diago + offdia * diff;
  sym_add(acc + SC_WT, g, offdia / q2);
}

// The terms of stored frequency p = (kx, position yi, position zi), whose
// natural indices are (kx, ky, kz), added to acc[NSC].  st[sp] is species
// sp's structure factor there, without the B-spline factor b1 b2 b3.
template <typename T>
HD void stress_point(const SlotDev& s, const StressArgs& sa, long long p, int kx, int ky, int kz,
                     const cx<double>* st, double* acc) {
  const int n1 = s.n1, n2 = s.n2, n3 = s.n3;
  const int m2 = signed_freq(ky, n2), m3 = signed_freq(kz, n3);
  const double* R = s.recip;
  double g[3], ge[3];
  for (int r = 0; r < 3; ++r) g[r] = R[r] * kx + R[3 + r] * m2 + R[6 + r] * m3;
  const bool wgc = s.kinetic == KIN_WGC;  // WGC fields: rho, sqrt(rho), then the alpha and beta triples
  const cx<double> F0 = spec_at<T>(s, 0, p), Fs = spec_at<T>(s, wgc ? 1 : 2, p);
  // vW
  const bool edge = kx == 0 || ((n1 % 2) == 0 && kx == n1 / 2);
  if (edge) {
    const int e1 = 0;
    const int e2 = ((n2 % 2) == 0 && ky == n2 / 2) ? 0 : m2;
    const int e3 = ((n3 % 2) == 0 && kz == n3 / 2) ? 0 : m3;
    for (int r = 0; r < 3; ++r) ge[r] = R[r] * e1 + R[3 + r] * e2 + R[6 + r] * e3;
  } else {
    for (int r = 0; r < 3; ++r) ge[r] = g[r];
  }
  sym_add(acc + SC_VW, ge, (edge ? 1.0 : 2.0) * (Fs.x * Fs.x + Fs.y * Fs.y));
  if (!stress_mask(kx, ky, kz, n1, n2, n3)) return;
  const double q2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
  const double q = sqrt(q2);
  // Hartree
  sym_add(acc + SC_H, g, (F0.x * F0.x + F0.y * F0.y) / (q2 * q2));
  const double eta = q / (2.0 * sa.kf);
  if (wgc) {
    stress_wgc_point<T>(s, sa, p, g, q2, eta, acc);
  } else {  // WT
    const cx<double> Fb = spec_at<T>(s, 1, p);
    const cx<double> Fa = s.nf > 3 ? spec_at<T>(s, 3, p) : Fb;
    const double diff = -eta * wt_g_prime(eta, s.mu) * (Fa.x * Fb.x + Fa.y * Fb.y);
    sym_add(acc + SC_WT, g, diff / q2);
    acc[SC_WTTR] += diff;
  }
  // ion-electron
  if (sa.nion > 0) {
    double tr = 0.0, ti = 0.0;
#pragma unroll
    for (int sp = 0; sp < MAX_SPECIES; ++sp) {
      if (sp >= s.ion.nspec) break;
      const double v = psp_diff(s.ion, sp, q) / q;
      tr += st[sp].x * v;
      ti += st[sp].y * v;
    }
    const cx<double> bb = cmul(cmul(s.ion.b1[kx], s.ion.b2[ky]), s.ion.b3[kz]);
    const cx<double> sf = cmul(bb, mk<double>(tr * s.inv_n, ti * s.inv_n));
    sym_add(acc + SC_IE, g, F0.x * sf.x - F0.y * sf.y);
  }
}

// Block b of nblk: the rows (kx, yi) r = b, b + nblk, ..., their zi spread over
// the threads.  The structure factor of a row is a contraction over the ions,
// sum_i (A_x A_y)_i A_z(i, kz): the products A_x A_y of a row go to shared
// memory once (chunks of STRESS_CHUNK ions), so a frequency costs four
// multiply-adds an ion instead of two complex products and the table loads
// (108 ions, 72^3: see k_stress).
constexpr int STRESS_CHUNK = 256;
template <typename T>
HD void stress_block(const SlotDev& s, const StressArgs& sa, int b, int nblk, int tid, int nthr, cx<double>* prod,
                     double* red, double* out) {
  const int n2 = s.n2, n3 = s.n3, rows = s.k1 * n2, L = s.k1 + n2 + n3;
  double acc[NSC];
  for (int k = 0; k < NSC; ++k) acc[k] = 0.0;
  for (int r = b; r < rows; r += nblk) {
    const int kx = r / n2, yi = r - kx * n2, ky = sa.permy[yi];
    for (int z0 = 0; z0 < n3; z0 += nthr) {
      const int zi = z0 + tid, kz = zi < n3 ? sa.permz[zi] : 0;
      cx<double> st[MAX_SPECIES];
#pragma unroll
      for (int sp = 0; sp < MAX_SPECIES; ++sp) st[sp] = mk<double>(0.0, 0.0);
      for (int i0 = 0; i0 < sa.nion; i0 += STRESS_CHUNK) {
        const int ni = sa.nion - i0 < STRESS_CHUNK ? sa.nion - i0 : STRESS_CHUNK;
        BLOCK_SYNC();
        for (int i = tid; i < ni; i += nthr) {
          const cx<double>* A = sa.sf + (size_t)(i0 + i) * L;
          prod[i] = cmul(A[kx], A[s.k1 + ky]);
        }
        BLOCK_SYNC();
        const cx<double>* az = sa.sf + (size_t)i0 * L + s.k1 + n2 + kz;
#pragma unroll
        for (int sp = 0; sp < MAX_SPECIES; ++sp) {
          if (sp >= s.ion.nspec) break;
          if (s.ion.nspec == 1) {
#pragma unroll 8
            for (int i = 0; i < ni; ++i) {
              const cx<double> x = cmul(prod[i], az[(size_t)i * L]);
              st[sp].x += x.x;
              st[sp].y += x.y;
            }
            break;
          }
          for (int i = 0; i < ni; ++i) {
            if (sa.species[i0 + i] != sp) continue;
            const cx<double> x = cmul(prod[i], az[(size_t)i * L]);
            st[sp].x += x.x;
            st[sp].y += x.y;
          }
        }
      }
      if (zi < n3) stress_point<T>(s, sa, ((long long)kx * n3 + zi) * n2 + yi, kx, ky, kz, st, acc);
    }
  }
  BLOCK_SYNC();
  block_sum<NSC>(red, acc, tid, nthr, out);
}

// Sum of rho * v_xc (Perdew-Zunger LDA, in FP64) over the points of block b
// of nblk; thread 0 writes out[0].
template <typename T>
HD void rho_vxc_block(const T* rho, long long n, int b, int nblk, int tid, int nthr, double* red, double* out) {
  double acc = 0.0;
  const long long stride = (long long)nblk * nthr;
  for (long long k = (long long)b * nthr + tid; k < n; k += stride) {
    const double r = (double)rho[k];
    const double r13 = cbrt(r);
    double vxc, exc;
    const double rs = 0.62035049089940009 / r13;
    lda_point<double>(r, r13, rs, sqrt(rs), vxc, exc);
    acc += r * vxc;
  }
  block_sum<1>(red, &acc, tid, nthr, out);
}

// Sum of v over block b of nblk (strided like rho_vxc_block); thread 0 writes out[0].
template <typename T>
HD void sum_block(const T* v, long long n, int b, int nblk, int tid, int nthr, double* red, double* out) {
  double acc = 0.0;
  const long long stride = (long long)nblk * nthr;
  for (long long k = (long long)b * nthr + tid; k < n; k += stride) acc += (double)v[k];
  block_sum<1>(red, &acc, tid, nthr, out);
}

#if !defined(OFDFT_EMU)
__global__ void __launch_bounds__(128) k_stress_sf(const SlotDev* sd, const IonStencil* st, cx<double>* sf) {
  const SlotDev& s = *sd;
  const int L = s.k1 + s.n2 + s.n3;
  for (int w = threadIdx.x; w < L; w += blockDim.x)
    sf[(size_t)blockIdx.x * L + w] = stress_sf_entry(s, st[blockIdx.x], w);
}
template <typename T>
__global__ void __launch_bounds__(128) k_stress(const SlotDev* sd, StressArgs sa, double* out) {
  __shared__ double red[NSC * 128];
  __shared__ cx<double> prod[STRESS_CHUNK];
  stress_block<T>(*sd, sa, blockIdx.x, gridDim.x, threadIdx.x, blockDim.x, prod, red,
                  out + (size_t)NSC * blockIdx.x);
}
template <typename T>
__global__ void __launch_bounds__(256) k_rho_vxc(const T* rho, long long n, double* out) {
  __shared__ double red[256];
  rho_vxc_block<T>(rho, n, blockIdx.x, gridDim.x, threadIdx.x, blockDim.x, red, out + blockIdx.x);
}
template <typename T>
__global__ void __launch_bounds__(256) k_sum(const T* v, long long n, double* out) {
  __shared__ double red[256];
  sum_block<T>(v, n, blockIdx.x, gridDim.x, threadIdx.x, blockDim.x, red, out + blockIdx.x);
}
template <typename T>
__global__ void __launch_bounds__(256) k_scale(T* v, long long n, double f) {
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    v[k] = (T)((double)v[k] * f);
}
#endif

}  // namespace ofdft
