// lut_batch.cuh -- the table kernels (lut.cuh) on a work list of stripes.
// Instantiated per element width in lut_e1.cu, lut_e2.cu, lut_e4.cu and lut_e8.cu.
#pragma once
#include "lut_single.cuh"

namespace fgfc {

// Persistent CTAs claim items (job, part) from a counter: entries of a list, or,
// where every job has `each` parts, positions in a list of jobs. Part p of a job's
// `parts` takes its tiles p, p + parts, ..., part `parts` its edges. The next
// item is claimed before the current one is worked on, and the tables are
// refilled (a few KiB) only where the plan changes. Sources past kc (one fill's
// limit) accumulate in further rounds over the same tiles.
template <int E, int LEV, int W, int MODE>
__global__ void __launch_bounds__(kLutThreads, lut_min_ctas<E, LEV, W, MODE>())
    lut_batch_kernel(const BatchDesc* __restrict__ jobs, const uint64_t* __restrict__ ptrs,
                     const void* __restrict__ items, uint32_t each, uint32_t nitems, uint32_t* counter, uint32_t kc) {
  using L = Lut<E, LEV>;
  using S = LutSmem<L::NV, W>;
  __shared__ LutShared sh;
  __shared__ LutBatchJob s_job;
  __shared__ uint32_t s_item;
  const uint32_t* resident = nullptr;
  uint32_t next = blockIdx.x;
  for (;;) {
    if (threadIdx.x == 0) s_item = next;
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= nitems) break;
    if (threadIdx.x == 0) next = gridDim.x + atomicAdd(counter, 1u);
    uint2 wi;
    if (each)
      wi = make_uint2(static_cast<const uint32_t*>(items)[it / each], it % each);
    else
      wi = static_cast<const uint2*>(items)[it];
    const LutBatchJob* jp = &jobs[wi.x].lut;
    const uint32_t k = jp->g.k;
    for (uint32_t t0 = 0; t0 < k; t0 += kc) {
      const uint32_t kk = min(kc, k - t0);
      if (t0) __syncthreads();  // the previous round is done with tables and pointers
      const uint32_t* img = jp->img + static_cast<size_t>(t0) * L::NV * W * 8;
      for (uint32_t i = threadIdx.x; i < kk; i += blockDim.x)
        sh.src[i] = reinterpret_cast<const uint8_t*>(ptrs[jp->src_idx + t0 + i]);
      for (uint32_t i = threadIdx.x; i < jp->g.nrows; i += blockDim.x)
        sh.dst[i] = reinterpret_cast<uint8_t*>(ptrs[jp->dst_idx + i]);
      if (threadIdx.x == 0) {
        s_job = *jp;
        s_job.g.k = kk;
        if (t0) s_job.g.ovr = 0;
      }
      if (img != resident) {
        lut_fill<L, W>(img, kk);
        resident = img;
      }
      __syncthreads();
      const bool ovr = s_job.g.ovr != 0, fp = s_job.fp != 0;
      if (wi.y < s_job.parts) {
        lut_run<L, LEV, W, MODE>(s_job.g, sh, wi.y, s_job.parts, ovr, fp);
      } else {
        uint8_t* stage = g_smem + kk / 3u * S::block3 + kk % 3u * S::block1;
        lut_edges<L, LEV, W, MODE>(s_job.g, sh, stage, ovr, fp);
      }
    }
    __syncthreads();  // done with tables, pointers and s_item
  }
}

template <int E, int LEV, int W>
LutBatchKernel lut_batch_lw(int mode) {
  LutBatchKernel b;
  b.fn = mode == kAligned   ? lut_batch_kernel<E, LEV, W, kAligned>
         : mode == kRowsOff ? lut_batch_kernel<E, LEV, W, kRowsOff>
                            : lut_batch_kernel<E, LEV, W, kAnyOff>;
  b.ctas = mode == kAligned   ? lut_min_ctas<E, LEV, W, kAligned>()
           : mode == kRowsOff ? lut_min_ctas<E, LEV, W, kRowsOff>()
                              : lut_min_ctas<E, LEV, W, kAnyOff>();
  return b;
}

}  // namespace fgfc
