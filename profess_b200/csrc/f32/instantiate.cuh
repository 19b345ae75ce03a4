// What the units pass_*_f32.cu instantiate: a kernel, or in the host emulation
// its block function.
#pragma once
#include "passes.cuh"

#if !defined(OFDFT_EMU)
#include <cuda_runtime.h>

namespace ofdft {
namespace f32 {

// Minimum resident 256-thread blocks per SM of the x and split y/z passes (it
// caps the registers at 65536 / (256 * minb)).
constexpr int PASS_MINB = 4;
template <typename T, int KS> __global__ void __launch_bounds__(256, PASS_MINB) k_xfwd(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  xfwd_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}
template <typename T> __global__ void __launch_bounds__(256, PASS_MINB) k_ypass(Args<T> a, int dir) {
  extern __shared__ __align__(16) char sm[];
  ypass_block<T>(a, blockIdx.x, threadIdx.x, blockDim.x, sm, dir);
}
template <typename T, int KS> __global__ void __launch_bounds__(256, PASS_MINB) k_zpass(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  zpass_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}
// Fused y-z pass: 256-thread blocks, up to three per SM; 512-thread blocks, one
// per SM, for larger planes.
template <typename T, int NT, int KS>
__global__ void __launch_bounds__(NT, NT == 256 ? 3 : 1) k_yzpass(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  yzpass_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}
template <typename T, int KS> __global__ void __launch_bounds__(256, PASS_MINB) k_xinv(Args<T> a) {
  extern __shared__ __align__(16) char sm[];
  xinv_block<T, KS>(a, blockIdx.x, threadIdx.x, blockDim.x, sm);
}

}  // namespace f32
}  // namespace ofdft
#endif
