#define OFDFT_INSTANTIATE
#include "kernels.cuh"
namespace ofdft {
OFDFT_YZG_KERNELS(double, )
}
