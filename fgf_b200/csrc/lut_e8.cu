// lut_e8.cu -- the table kernels (lut.cuh) of the 8-byte fields.
#include "lut_batch.cuh"

namespace fgfc {

cudaError_t lut_launch_e8(int lev, int w, LutArgs& a, cudaStream_t s, bool unal, bool edges_only) {
  if (lev == 1 && w == 1) return lut_launch_lw<8, 1, 1>(a, s, unal, edges_only);
  if (lev == 2 && w == 1) return lut_launch_lw<8, 2, 1>(a, s, unal, edges_only);
  if (lev == 3 && w == 1) return lut_launch_lw<8, 3, 1>(a, s, unal, edges_only);
  return cudaErrorInvalidValue;
}

LutBatchKernel lut_batch_e8(int lev, int w, bool unal) {
  if (lev == 1 && w == 1) return lut_batch_lw<8, 1, 1>(unal);
  if (lev == 2 && w == 1) return lut_batch_lw<8, 2, 1>(unal);
  if (lev == 3 && w == 1) return lut_batch_lw<8, 3, 1>(unal);
  return LutBatchKernel{};
}

}  // namespace fgfc
