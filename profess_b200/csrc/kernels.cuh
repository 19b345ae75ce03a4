// The kernels of the FP64 evaluation passes (FP32: f32/kernels.cuh).  They hold most of the library's code
// (every radix of every stage), so each is instantiated in a translation unit
// of its own (pass_*.cu): the units compile side by side, and a unit's code
// does not depend on what else is compiled with it.  engine.cu sees them as
// extern templates.
#pragma once
#include "passes.cuh"

#if !defined(OFDFT_EMU)
#include <cuda_runtime.h>

namespace ofdft {

// Minimum resident 256-thread blocks per SM of the kernels (they cap the
// registers at 65536 / (256 * minb)): three, but for the z pass of a WGC cell,
// which keeps three columns in registers (160 x 160 x 256: 336 us with two
// blocks, 384 with three; 100 x 100 x 128: 98 and 112; WT z pass: 180^3 136 and 119,
// 512 x 128 x 256 383 and 325; y pass: 100 x 100 x 128 WGC 53 and 44, 512 x 128 x
// 256 249 and 223, 180^3 103 and 104).
constexpr int X_MINB = 3, Y_MINB = 3, YZ_MINB = 3;
constexpr int z_minb(int ks) { return ks == KS_WGC ? 2 : 3; }
template <typename T, int KS> __global__ void __launch_bounds__(256, X_MINB) k_xfwd(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  xfwd_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}
template <typename T> __global__ void __launch_bounds__(256, Y_MINB) k_ypass(Args<T> a, int dir) {
  extern __shared__ __align__(16) char sm[];
  ypass_block<T>(a, blockIdx.x, threadIdx.x, blockDim.x, sm, dir);
}
template <typename T, int KS> __global__ void __launch_bounds__(256, z_minb(KS)) k_zpass(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  zpass_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}
// Fused y-z pass: 256-thread blocks, up to three per SM, for planes up to
// YZ_SMEM_SMALL; 512-thread blocks, one per SM, for larger planes.
template <typename T, int NT, int KS>
__global__ void __launch_bounds__(NT, NT < 512 ? YZ_MINB : 1) k_yzpass(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  yzpass_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}
template <typename T, int KS> __global__ void __launch_bounds__(256, X_MINB) k_xinv(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  xinv_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}

#define OFDFT_XFWD_KERNELS(T, X)                                      \
  X template __global__ void k_xfwd<T, KS_WT>(Args<T>);               \
  X template __global__ void k_xfwd<T, KS_WGC>(Args<T>);
#define OFDFT_XINV_KERNELS(T, X)                                      \
  X template __global__ void k_xinv<T, KS_WT>(Args<T>);               \
  X template __global__ void k_xinv<T, KS_WGC>(Args<T>);
#define OFDFT_YZ_KERNELS(T, X)                                        \
  X template __global__ void k_yzpass<T, 256, KS_WT>(Args<T>);        \
  X template __global__ void k_yzpass<T, 512, KS_WT>(Args<T>);
#define OFDFT_YZG_KERNELS(T, X)                                       \
  X template __global__ void k_yzpass<T, 256, KS_WGC>(Args<T>);       \
  X template __global__ void k_yzpass<T, 512, KS_WGC>(Args<T>);
#define OFDFT_SPLIT_KERNELS(T, X)                                     \
  X template __global__ void k_ypass<T>(Args<T>, int);                \
  X template __global__ void k_zpass<T, KS_WT>(Args<T>);              \
  X template __global__ void k_zpass<T, KS_WGC>(Args<T>);
#define OFDFT_PASS_KERNELS(T, X)                                      \
  OFDFT_XFWD_KERNELS(T, X)                                            \
  OFDFT_XINV_KERNELS(T, X)                                            \
  OFDFT_YZ_KERNELS(T, X)                                              \
  OFDFT_YZG_KERNELS(T, X)                                             \
  OFDFT_SPLIT_KERNELS(T, X)

#if !defined(OFDFT_INSTANTIATE)
OFDFT_PASS_KERNELS(double, extern)
#endif

}  // namespace ofdft
#endif
