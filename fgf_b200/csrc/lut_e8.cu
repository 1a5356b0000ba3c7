// lut_e8.cu -- the table kernels (lut.cuh) of the 8-byte fields.
#include "lut_batch.cuh"

namespace fgfc {

cudaError_t lut_launch_e8(int lev, int w, LutArgs& a, cudaStream_t s, int mode) {
  if (lev == 1 && w == 1) return lut_launch_lw<8, 1, 1>(a, s, mode);
  if (lev == 2 && w == 1) return lut_launch_lw<8, 2, 1>(a, s, mode);
  if (lev == 3 && w == 1) return lut_launch_lw<8, 3, 1>(a, s, mode);
  return cudaErrorInvalidValue;
}

LutBatchKernel lut_batch_e8(int lev, int w, int mode) {
  if (lev == 1 && w == 1) return lut_batch_lw<8, 1, 1>(mode);
  if (lev == 2 && w == 1) return lut_batch_lw<8, 2, 1>(mode);
  if (lev == 3 && w == 1) return lut_batch_lw<8, 3, 1>(mode);
  return LutBatchKernel{};
}

}  // namespace fgfc
