#define OFDFT_INSTANTIATE
#include "kernels.cuh"
namespace ofdft {
OFDFT_XINV_KERNELS(double, )
}
