#include "f32/kernels.cuh"
namespace ofdft {
template __global__ void k_yzpass<float, 256, KS_WT>(Args<float>);
template __global__ void k_yzpass<float, 512, KS_WT>(Args<float>);
}
