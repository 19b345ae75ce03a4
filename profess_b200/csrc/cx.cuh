// Basic device helpers shared by all kernels of the density-solve engine.
//
// Every kernel body is written as a "block function": a __host__ __device__
// function that receives the block index, the thread index and the block size
// explicitly and synchronises only through BLOCK_SYNC().  On the device it runs
// inside a __global__ wrapper; in the host-emulation build (OFDFT_EMU, a test
// harness) the same body runs once per block with a single thread, so the block
// function must do all per-thread work in strided loops and keep no per-thread
// register state across a BLOCK_SYNC().
#pragma once
#include <cstdint>
#include <cmath>
#include <cstring>

#if defined(__CUDACC__)
#define HD __host__ __device__ __forceinline__
#define HDNI __host__ __device__
#define HDC __host__ __device__ constexpr
#else
#define HD inline
#define HDNI
#define HDC constexpr
#endif

#if defined(__CUDA_ARCH__)
#define BLOCK_SYNC() __syncthreads()
#else
#define BLOCK_SYNC() ((void)0)
#endif

namespace ofdft {

template <typename T>
struct alignas(2 * sizeof(T)) cx {
  T x, y;
};

template <typename T> HD cx<T> mk(T a, T b) { cx<T> r; r.x = a; r.y = b; return r; }
template <typename T> HD cx<T> operator+(cx<T> a, cx<T> b) { return mk<T>(a.x + b.x, a.y + b.y); }
template <typename T> HD cx<T> operator-(cx<T> a, cx<T> b) { return mk<T>(a.x - b.x, a.y - b.y); }
template <typename T> HD cx<T> operator*(cx<T> a, T s) { return mk<T>(a.x * s, a.y * s); }
template <typename T> HD cx<T> cmul(cx<T> a, cx<T> b) {
  return mk<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename T> HD cx<T> conj(cx<T> a) { return mk<T>(a.x, -a.y); }
// multiply by dir * i  (dir = +1 or -1)
template <typename T> HD cx<T> mul_i(cx<T> a, int dir) {
  return dir > 0 ? mk<T>(-a.y, a.x) : mk<T>(a.y, -a.x);
}

// Precision-generic math wrappers (float versions map to the float library calls).
HD double m_sqrt(double v) { return sqrt(v); }
HD float m_sqrt(float v) { return sqrtf(v); }
HD float m_cbrt(float v) { return cbrtf(v); }
HD double m_pow(double a, double b) { return pow(a, b); }
HD float m_pow(float a, float b) { return powf(a, b); }
// The power as a call, for a rare case: its code does not take registers from
// the common one.
#if defined(__CUDA_ARCH__)
__device__ __noinline__ inline double m_pow_call(double a, double b) { return pow(a, b); }
#else
HD double m_pow_call(double a, double b) { return pow(a, b); }
#endif
HD double m_log(double v) { return log(v); }
HD float m_log(float v) { return logf(v); }
#if defined(__CUDA_ARCH__)
HD float m_rcbrt(float v) { return rcbrtf(v); }
HD double m_rsqrt(double v) { return rsqrt(v); }
#else
HD float m_rcbrt(float v) { return 1.0f / cbrtf(v); }
HD double m_rsqrt(double v) { return 1.0 / sqrt(v); }
#endif

// a^(-1/3) and, in m_icbrt2, a^(-2/3) of a in [1e-30, 1e30] (icbrt_out says when
// it is not: the caller then takes m_icbrt_any, once for a whole group of
// values, so that the fast path is free of branches).  A single-precision seed
// y (exp2 of -log2(a)/3 of the float with a's leading bits) and one step of the
// series of (1 - e)^(-1/3) and (1 - e)^(-2/3) in e = 1 - a y^3 on y and y^2, which
// is exact: a seed has 24 bits.  The seed's error is about 1e-6 near a = 1 and
// grows with |log2 a| to 3e-6 at the ends of the range; the first term left out,
// 35/243 e^4 and 110/243 e^4, is below 1e-20.  What remains is the rounding of a y in
// e and of the result, as in rcbrt.  rho^(-1/3) as the square of rho^(-1/6) has twice that
// error, and its cube, 1/rho, six times (RMS error of rho^(-1/3) over [1e-5, 10]
// 1.1e-16 that way, 5e-17 by the second series and by rcbrt).
HD bool icbrt_out(double a) { return !(a >= 1e-30 && a <= 1e30); }
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ double icbrt_seed(double a) {
  const int h = ((__double2hiint(a) - 0x38000000) << 3) | (int)((unsigned)__double2loint(a) >> 29);
  float s = -0.333333343f * __log2f(__int_as_float(h));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(s));
  const int b = __float_as_int(s);
  return __hiloint2double((b >> 3) + 0x38000000, b << 29);
}
#endif
HD double m_icbrt(double a) {
#if defined(__CUDA_ARCH__)
  const double y = icbrt_seed(a);
  const double e = fma(-(a * y), y * y, 1.0);
  return fma(y * e, fma(e, fma(e, 14.0 / 81.0, 2.0 / 9.0), 1.0 / 3.0), y);
#else
  return 1.0 / cbrt(a);
#endif
}
HD void m_icbrt2(double a, double& y1, double& y2) {
#if defined(__CUDA_ARCH__)
  const double y = icbrt_seed(a), s = y * y;
  const double e = fma(-(a * y), s, 1.0);
  y1 = fma(y * e, fma(e, fma(e, 14.0 / 81.0, 2.0 / 9.0), 1.0 / 3.0), y);
  y2 = fma(s * e, fma(e, fma(e, 40.0 / 81.0, 5.0 / 9.0), 2.0 / 3.0), s);
#else
  y1 = 1.0 / cbrt(a);
  y2 = 1.0 / cbrt(a * a);
#endif
}
#if defined(__CUDA_ARCH__)
__device__ __noinline__ inline double m_icbrt_any(double a) { return rcbrt(a); }
#else
HD double m_icbrt_any(double a) { return 1.0 / cbrt(a); }
#endif

}  // namespace ofdft
