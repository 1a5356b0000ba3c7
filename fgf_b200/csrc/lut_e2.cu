// lut_e2.cu -- the table kernels (lut.cuh) of the 2-byte fields.
#include "lut_batch.cuh"

namespace fgfc {

cudaError_t lut_launch_e2(int lev, int w, LutArgs& a, cudaStream_t s, int mode) {
  if (lev == 0 && w == 1) return lut_launch_lw<2, 0, 1>(a, s, mode);
  if (lev == 0 && w == 2) return lut_launch_lw<2, 0, 2>(a, s, mode);
  if (lev == 0 && w == 3) return lut_launch_lw<2, 0, 3>(a, s, mode);
  if (lev == 0 && w == 4) return lut_launch_lw<2, 0, 4>(a, s, mode);
  if (lev == 1 && w == 1) return lut_launch_lw<2, 1, 1>(a, s, mode);
  if (lev == 1 && w == 2) return lut_launch_lw<2, 1, 2>(a, s, mode);
  return cudaErrorInvalidValue;
}

LutBatchKernel lut_batch_e2(int lev, int w, int mode) {
  if (lev == 0 && w == 1) return lut_batch_lw<2, 0, 1>(mode);
  if (lev == 0 && w == 2) return lut_batch_lw<2, 0, 2>(mode);
  if (lev == 0 && w == 3) return lut_batch_lw<2, 0, 3>(mode);
  if (lev == 0 && w == 4) return lut_batch_lw<2, 0, 4>(mode);
  if (lev == 1 && w == 1) return lut_batch_lw<2, 1, 1>(mode);
  if (lev == 1 && w == 2) return lut_batch_lw<2, 1, 2>(mode);
  return LutBatchKernel{};
}

}  // namespace fgfc
