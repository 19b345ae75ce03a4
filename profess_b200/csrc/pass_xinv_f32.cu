#include "f32/instantiate.cuh"
namespace ofdft {
namespace f32 {
#if defined(OFDFT_EMU)
template void xinv_block<float, KS_WT>(const Args<float>&, int, int, int, char*);
template void xinv_block<float, KS_WGC>(const Args<float>&, int, int, int, char*);
#else
template __global__ void k_xinv<float, KS_WT>(Args<float>);
template __global__ void k_xinv<float, KS_WGC>(Args<float>);
#endif
}  // namespace f32
}  // namespace ofdft
