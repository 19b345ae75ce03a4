#include "f32/instantiate.cuh"
namespace ofdft {
namespace f32 {
#if defined(OFDFT_EMU)
template void yzpass_block<float, KS_WT>(const Args<float>&, int, int, int, char*);
#else
template __global__ void k_yzpass<float, 256, KS_WT>(Args<float>);
template __global__ void k_yzpass<float, 512, KS_WT>(Args<float>);
#endif
}  // namespace f32
}  // namespace ofdft
