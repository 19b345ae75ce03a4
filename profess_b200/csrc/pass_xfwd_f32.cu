#include "f32/kernels.cuh"
namespace ofdft {
template __global__ void k_xfwd<float, KS_WT>(Args<float>);
template __global__ void k_xfwd<float, KS_WGC>(Args<float>);
}
