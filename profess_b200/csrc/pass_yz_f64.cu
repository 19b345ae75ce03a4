#define OFDFT_INSTANTIATE
#include "kernels.cuh"
namespace ofdft {
OFDFT_YZ_KERNELS(double, )
}
