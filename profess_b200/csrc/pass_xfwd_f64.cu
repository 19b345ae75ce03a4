#define OFDFT_INSTANTIATE
#include "kernels.cuh"
namespace ofdft {
OFDFT_XFWD_KERNELS(double, )
}
