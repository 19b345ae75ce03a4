// The pass kernels of the FP32 slots, as engine.cu sees them (pass_*_f32.cu
// instantiates them from passes.cuh); in the host emulation, their block
// functions.
#pragma once
#include "shape.cuh"

namespace ofdft {
namespace f32 {

#if defined(OFDFT_EMU)
template <typename T, int KS> void xfwd_block(const Args<T>& a, int bid, int tid, int nthr, char* smem);
template <typename T> void ypass_block(const Args<T>& a, int bid, int tid, int nthr, char* smem, int dir);
template <typename T, int KS> void zpass_block(const Args<T>& a, int bid, int tid, int nthr, char* smem);
template <typename T, int KS> void yzpass_block(const Args<T>& a, int bid, int tid, int nthr, char* smem);
template <typename T, int KS> void xinv_block(const Args<T>& a, int bid, int tid, int nthr, char* smem);
#else
template <typename T, int KS> __global__ void k_xfwd(Args<T> a);
template <typename T> __global__ void k_ypass(Args<T> a, int dir);
template <typename T, int KS> __global__ void k_zpass(Args<T> a);
template <typename T, int NT, int KS> __global__ void k_yzpass(Args<T> a);
template <typename T, int KS> __global__ void k_xinv(Args<T> a);
#endif

}  // namespace f32
}  // namespace ofdft
