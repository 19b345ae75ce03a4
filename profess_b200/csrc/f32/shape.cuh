// Shared memory of the FP32 x passes (the engine sizes their tasks by it).
#pragma once
#include "../pass_common.cuh"

namespace ofdft {
namespace f32 {

// Shared memory of an x-inverse task with nfb transformed fields (or ion
// species) and nb row pairs, elements of esz bytes: the transform buffer,
// then the reduction scratch.
HD size_t xinv_smem(int n1, int nfb, int nb, size_t esz) {
  return align16((size_t)nfb * nb * n1 * 2 * esz) + NCH * 33 * sizeof(double);
}

// Shared memory of an x-forward task: the transform buffer, then the task's
// rows of the two evaluation inputs.
HD size_t xfwd_stage_offset(int n1, int nfb, int nb, size_t esz) {
  return align16((size_t)nfb * nb * n1 * 2 * esz);
}
HD size_t xfwd_smem(int n1, int nfb, int nb, size_t esz) {
  return xfwd_stage_offset(n1, nfb, nb, esz) + 2 * align16((size_t)2 * nb * n1 * esz);
}

}  // namespace f32
}  // namespace ofdft
