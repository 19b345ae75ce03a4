#define OFDFT_INSTANTIATE
#include "kernels.cuh"
namespace ofdft {
OFDFT_SPLIT_KERNELS(double, )
}
