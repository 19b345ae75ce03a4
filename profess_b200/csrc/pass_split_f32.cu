#include "f32/kernels.cuh"
namespace ofdft {
template __global__ void k_ypass<float>(Args<float>, int);
template __global__ void k_zpass<float, KS_WT>(Args<float>);
template __global__ void k_zpass<float, KS_WGC>(Args<float>);
}
