// Ewald sum of point charges on the device (EwaldEnergy / EwaldForces,
// Source/Ewald.f90:465-1193): the splitting and cut-offs of the host sum
// (ewald_par in setup.cuh), in three launches:
//   phases      - the one-dimensional phases exp(2 pi i m f_a) of every ion,
//                 axis a and index |m| <= ng[a];
//   sums        - real space, block i: every partner and image of ion i
//                 inside the cut-off; and reciprocal space, block (m1, m2) of
//                 the half space m1 >= 0: S(G) = sum_i z_i exp(i G.R_i) of
//                 that row of G and the row's energy;
//   rec. forces - block i: the force on ion i from every stored S(G).
// Each block adds its threads' partials in a fixed tree and the host adds the
// blocks in index order, so the result does not depend on scheduling.
//
// What bounds it: the FP64 pipe (erfc and exp of a pair, 4 multiply-adds of a
// phase product).  The work per block is therefore cut to what the cut-offs
// leave: partner differences are wrapped to [-1/2, 1/2) first, so an axis
// needs the images |m| <= rcut / height + 1/2 and not every image two cells
// could reach (500 ions: 27 instead of 343 images a pair), and a phase
// exp(i G.R) is the product of three table entries instead of a sine and a
// cosine of its own (the angles m f are reduced exactly before the sine, so a
// product is closer to exact than the direct sine of a large angle).  Energy
// and forces of 256 / 500 / 1152 ions: 455 / 1280 / 3700 us of kernels with a
// sine and cosine per (ion, G) and every image -> 98 / 154 / about 450 us.
#pragma once

#include "cx.cuh"
#include "setup.cuh"

namespace ofdft {

// Fixed-order sum of K values per thread over the block; thread 0 writes
// out[0..K-1].  red holds K * nthr doubles.
template <int K>
HD void block_sum(double* red, const double* v, int tid, int nthr, double* out) {
  for (int k = 0; k < K; ++k) red[K * tid + k] = v[k];
  BLOCK_SYNC();
  for (int st = 1; st < nthr; st *= 2) {
    if ((tid % (2 * st)) == 0 && tid + st < nthr)
      for (int k = 0; k < K; ++k) red[K * tid + k] += red[K * (tid + st) + k];
    BLOCK_SYNC();
  }
  if (tid == 0)
    for (int k = 0; k < K; ++k) out[k] = red[k];
}

// a[0..5] += w * (upper triangle of g g^T).
HD void sym_add(double* a, const double* g, double w) {
  a[0] += w * g[0] * g[0];
  a[1] += w * g[0] * g[1];
  a[2] += w * g[0] * g[2];
  a[3] += w * g[1] * g[1];
  a[4] += w * g[1] * g[2];
  a[5] += w * g[2] * g[2];
}

// Lane, lanes, warp and warps of a thread (the host emulation's block is one
// thread: one warp of one lane), and the fixed-order sum over a warp's lanes
// (the total is in lane 0).
struct Lanes {
  int lane, nl, warp, nw;
  HD Lanes(int tid, int nthr) : lane(tid & 31), nl(nthr < 32 ? nthr : 32), warp(tid >> 5), nw((nthr + 31) >> 5) {}
};
HD double warp_sum(double x) {
#if defined(__CUDA_ARCH__)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
#endif
  return x;
}

HD int ewald_nm(const EwaldPar& p, int a) { return 2 * p.ng[a] + 1; }
// Blocks of the reciprocal sum: the rows (m1 >= 0, m2); each holds
// ewald_nm(p, 2) values of m3.
HD int ewald_rows(const EwaldPar& p) { return (p.ng[0] + 1) * ewald_nm(p, 1); }
HD int ewald_phases(const EwaldPar& p) { return (ewald_nm(p, 0) + ewald_nm(p, 1) + ewald_nm(p, 2)) * p.nion; }

// Table of the axis-a phases: entry (m, ion) at [(m + ng[a]) * nion + ion].
HD const cx<double>* ewald_axis(const EwaldPar& p, const cx<double>* tab, int a) {
  int off = 0;
  for (int b = 0; b < a; ++b) off += ewald_nm(p, b);
  return tab + (size_t)off * p.nion;
}

// Entry w of the phase table: exp(2 pi i m f), m f reduced to [-1/2, 1/2]
// with one rounding before the sine.
HD cx<double> ewald_phase(const EwaldPar& p, const double* frac, int w) {
  int m = w / p.nion, a = 0;
  const int i = w - m * p.nion;
  while (m >= ewald_nm(p, a)) m -= ewald_nm(p, a++);
  const double dm = (double)(m - p.ng[a]), f = frac[3 * i + a];
  const double t = fma(dm, f, -rint(dm * f));
  double sn, cs;
#if defined(__CUDA_ARCH__)
  sincospi(2.0 * t, &sn, &cs);
#else
  sn = std::sin(2.0 * PI_D * t);
  cs = std::cos(2.0 * PI_D * t);
#endif
  return mk<double>(cs, sn);
}

// f(j, d, r2) for every partner j and image of ion i inside the cut-off (d =
// R_j + L - R_i).  A work item is (partner, image along axes 0 and 1); the
// images along axis 2 are its inner loop.
template <class F>
HD void ewald_pairs(const EwaldPar& p, const double* frac, int i, int tid, int nthr, F f) {
  const int na = 2 * p.nw[0] + 1, nb = 2 * p.nw[1] + 1;
  const unsigned units = (unsigned)(na * nb) * (unsigned)p.nion;
  const double rc2 = p.rcut * p.rcut;
  const double fi[3] = {frac[3 * i], frac[3 * i + 1], frac[3 * i + 2]};
  for (unsigned w = tid; w < units; w += nthr) {
    const unsigned ab = w / (unsigned)p.nion;
    const int j = (int)(w - ab * (unsigned)p.nion);
    const int a = (int)(ab / (unsigned)nb);
    double s[3];
    for (int k = 0; k < 3; ++k) {
      const double df = frac[3 * j + k] - fi[k];
      s[k] = df - rint(df);
    }
    s[0] += (double)(a - p.nw[0]);
    s[1] += (double)((int)ab - a * nb - p.nw[1]);
    double e[3];
    for (int k = 0; k < 3; ++k) e[k] = p.A[k][0] * s[0] + p.A[k][1] * s[1];
    for (int c = -p.nw[2]; c <= p.nw[2]; ++c) {
      const double s2 = s[2] + (double)c;
      const double d[3] = {e[0] + p.A[0][2] * s2, e[1] + p.A[1][2] * s2, e[2] + p.A[2][2] * s2};
      const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
      if (r2 < 1e-24 || r2 >= rc2) continue;
      f(j, d, r2);
    }
  }
}

// out4 = (energy share of ion i, force on ion i) from the real-space sum.
HD void ewald_real_block(const EwaldPar& p, const double* frac, const double* z, int i, int tid, int nthr,
                         double* red, double* out4) {
  const double eta = p.eta, c2 = 2.0 * eta / sqrt(PI_D), zi = z[i];
  double v[4] = {0, 0, 0, 0};
  ewald_pairs(p, frac, i, tid, nthr, [&](int j, const double* d, double r2) {
    const double ri = m_rsqrt(r2), ec = erfc(eta * (r2 * ri)) * ri, zz = zi * z[j];
    v[0] += 0.5 * zz * ec;
    const double g = -zz * (ec + c2 * exp(-eta * eta * r2)) * (ri * ri);
    v[1] += g * d[0];
    v[2] += g * d[1];
    v[3] += g * d[2];
  });
  block_sum<4>(red, v, tid, nthr, out4);
}

// out7 = (0, the six components of sum 0.5 z_i z_j f'(r)/r d_a d_b) over the
// images and partners of ion i, f(r) = erfc(eta r)/r.
HD void ewald_real_stress_block(const EwaldPar& p, const double* frac, const double* z, int i, int tid, int nthr,
                                double* red, double* out7) {
  const double eta = p.eta, c2 = 2.0 * eta / sqrt(PI_D), zi = z[i];
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  ewald_pairs(p, frac, i, tid, nthr, [&](int j, const double* d, double r2) {
    const double ri = m_rsqrt(r2), ec = erfc(eta * (r2 * ri)) * ri;
    sym_add(v + 1, d, -0.5 * zi * z[j] * (ec + c2 * exp(-eta * eta * r2)) * (ri * ri));
  });
  block_sum<7>(red, v, tid, nthr, out7);
}

// G of reciprocal index (m1, m2, m3) and |G|^2.
HD double ewald_g(const EwaldPar& p, int m1, int m2, int m3, double* G) {
  for (int k = 0; k < 3; ++k) G[k] = 2.0 * PI_D * (p.inv[0][k] * m1 + p.inv[1][k] * m2 + p.inv[2][k] * m3);
  return G[0] * G[0] + G[1] * G[1] + G[2] * G[2];
}

// Row r = (m1, m2) of the half space: a warp takes one m3 at a time, its
// lanes the ions (in chunks of EWALD_CHUNK, whose products z e1 e2 are shared).
// S(G), times the force factor (4 pi / vol) exp(-G^2/4eta^2)/G^2 and the
// weight 2 of the conjugate half, goes to sf[r * nm3 + m3] (zero outside the
// cut-off and at G = 0); out[0] gets the row's energy and, with NOUT = 7,
// out[1..6] sum (2 pi / vol) exp(-G^2/4eta^2)/G^2 |S(G)|^2 2 (1/4eta^2 + 1/G^2) G_a G_b.
constexpr int EWALD_CHUNK = 256;
constexpr int EWALD_M3 = 128;  // m3 values of a row whose sums are kept between chunks
template <int NOUT>
HD void ewald_row_block(const EwaldPar& p, const cx<double>* tab, const double* z, int r, int tid, int nthr,
                        cx<double>* prod, cx<double>* part, double* red, cx<double>* sf, double* out) {
  const Lanes L(tid, nthr);
  const int n2 = ewald_nm(p, 1), nm3 = ewald_nm(p, 2);
  const int m1 = r / n2, m2 = r - m1 * n2 - p.ng[1];
  const cx<double>* e1 = ewald_axis(p, tab, 0) + (size_t)(m1 + p.ng[0]) * p.nion;
  const cx<double>* e2 = ewald_axis(p, tab, 1) + (size_t)(m2 + p.ng[1]) * p.nion;
  const cx<double>* e3 = ewald_axis(p, tab, 2);
  const double gc2 = p.gcut * p.gcut, e4 = 4.0 * p.eta * p.eta, wt = m1 > 0 ? 2.0 : 1.0;
  double v[NOUT];
  for (int k = 0; k < NOUT; ++k) v[k] = 0.0;
  for (int q0 = 0; q0 < nm3; q0 += EWALD_M3) {
    const int q1 = nm3 - q0 < EWALD_M3 ? nm3 : q0 + EWALD_M3;
    for (int i0 = 0; i0 < p.nion; i0 += EWALD_CHUNK) {
      const int ni = p.nion - i0 < EWALD_CHUNK ? p.nion - i0 : EWALD_CHUNK;
      BLOCK_SYNC();
      for (int i = tid; i < ni; i += nthr) prod[i] = cmul(e1[i0 + i], e2[i0 + i]) * z[i0 + i];
      BLOCK_SYNC();
      for (int q = q0 + L.warp; q < q1; q += L.nw) {
        const int m3 = q - p.ng[2];
        double G[3];
        const double g2 = ewald_g(p, m1, m2, m3, G);
        const bool in = g2 <= gc2 && !(m1 == 0 && m2 == 0 && m3 == 0);
        double sr = 0.0, si = 0.0;
        if (in) {
          const cx<double>* e = e3 + (size_t)q * p.nion + i0;
          for (int i = L.lane; i < ni; i += L.nl) {
            const cx<double> x = cmul(prod[i], e[i]);
            sr += x.x;
            si += x.y;
          }
        }
        sr = warp_sum(sr);
        si = warp_sum(si);
        if (L.lane != 0) continue;
        if (i0 > 0) {
          sr += part[q - q0].x;
          si += part[q - q0].y;
        }
        part[q - q0] = mk<double>(sr, si);
        if (i0 + ni < p.nion) continue;
        const double c = in ? wt * 2.0 * PI_D / p.vol * exp(-g2 / e4) / g2 : 0.0;
        sf[(size_t)r * nm3 + q] = mk<double>(2.0 * c * sr, 2.0 * c * si);
        if (!in) continue;
        const double en = c * (sr * sr + si * si);
        v[0] += en;
        if constexpr (NOUT == 7) sym_add(v + 1, G, en * 2.0 * (1.0 / e4 + 1.0 / g2));
      }
    }
  }
  BLOCK_SYNC();
  block_sum<NOUT>(red, v, tid, nthr, out);
}

// out[0..2] = reciprocal-space force on ion i from the stored S(G): a warp
// takes one row (m1, m2) at a time, its lanes m3 (whose phases stay in
// registers over the rows).
HD void ewald_recip_force_block(const EwaldPar& p, const cx<double>* tab, const double* z, const cx<double>* sf,
                                int i, int tid, int nthr, double* red, double* out) {
  const Lanes L(tid, nthr);
  const int n2 = ewald_nm(p, 1), nm3 = ewald_nm(p, 2), rows = ewald_rows(p);
  const cx<double>* e1 = ewald_axis(p, tab, 0) + (size_t)p.ng[0] * p.nion + i;
  const cx<double>* e2 = ewald_axis(p, tab, 1) + i;
  const cx<double>* e3 = ewald_axis(p, tab, 2) + i;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  for (int q = L.lane; q < nm3; q += L.nl) {
    const cx<double> z3 = e3[(size_t)q * p.nion];
    double b = 0.0;
    for (int r = L.warp; r < rows; r += L.nw) {
      const int m1 = r / n2, k2 = r - m1 * n2;
      const cx<double> e = cmul(cmul(e1[(size_t)m1 * p.nion], e2[(size_t)k2 * p.nion]), z3);
      const cx<double> S = sf[(size_t)r * nm3 + q];
      const double im = S.x * e.y - S.y * e.x;  // Im(conj(S) e^{i G R_i})
      a0 += (double)m1 * im;
      a1 += (double)(k2 - p.ng[1]) * im;
      b += im;
    }
    a2 += (double)(q - p.ng[2]) * b;
  }
  double v[3];
  for (int k = 0; k < 3; ++k) v[k] = 2.0 * PI_D * z[i] * (p.inv[0][k] * a0 + p.inv[1][k] * a1 + p.inv[2][k] * a2);
  block_sum<3>(red, v, tid, nthr, out);
}

#if !defined(OFDFT_EMU)
__global__ void __launch_bounds__(256) k_ewald_phase(EwaldPar p, const double* frac, cx<double>* tab) {
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < ewald_phases(p); w += gridDim.x * blockDim.x)
    tab[w] = ewald_phase(p, frac, w);
}
// Blocks [0, nion): real space; [nion, nion + rows): the reciprocal rows.
// NOUT = 4: energy and forces; 7: energy and stress.  out: NOUT values per block.
template <int NOUT>
__global__ void __launch_bounds__(128) k_ewald_sums(EwaldPar p, const double* frac, const double* z,
                                                    const cx<double>* tab, cx<double>* sf, double* out) {
  __shared__ double red[NOUT * 128];
  __shared__ cx<double> prod[EWALD_CHUNK], part[EWALD_M3];
  const int b = blockIdx.x;
  double* o = out + (size_t)NOUT * b;
  if (b >= p.nion)
    ewald_row_block<NOUT == 7 ? 7 : 1>(p, tab, z, b - p.nion, threadIdx.x, blockDim.x, prod, part, red, sf, o);
  else if constexpr (NOUT == 7)
    ewald_real_stress_block(p, frac, z, b, threadIdx.x, blockDim.x, red, o);
  else
    ewald_real_block(p, frac, z, b, threadIdx.x, blockDim.x, red, o);
}
__global__ void __launch_bounds__(128) k_ewald_recip_force(EwaldPar p, const cx<double>* tab, const double* z,
                                                           const cx<double>* sf, double* out) {
  __shared__ double red[3 * 128];
  ewald_recip_force_block(p, tab, z, sf, blockIdx.x, threadIdx.x, blockDim.x, red, out + 3 * (size_t)blockIdx.x);
}
#endif

}  // namespace ofdft
