// lut_batch.cuh -- the table kernels (lut.cuh) on a work list of stripes.
// Instantiated per element width in lut_e1.cu, lut_e2.cu, lut_e4.cu and lut_e8.cu.
#pragma once
#include "lut_single.cuh"

namespace fgfc {

// Persistent CTAs claim items (job, part) from a counter: entries of a list, or,
// where every job has `each` parts, positions in a list of jobs. Part p of a job's
// `parts` takes its tiles p, p + parts, ..., part `parts` its edges. The next item is
// claimed before the current one is worked on; where there is no more than one for
// every CTA they are taken by number, or the CTAs that start first would have the
// late ones' too (four Gf32 stripes of 1 MiB, (10,4), 64 items: 73 or 138 us). The
// tables are refilled (a few KiB) only where the plan changes. Sources past kc (one
// fill's limit) accumulate in further rounds over the same tiles.
template <int E, int LEV, int W, int MODE>
__global__ void __launch_bounds__(kLutThreads, lut_min_ctas<E, LEV, W, MODE>())
    lut_batch_kernel(const BatchDesc* __restrict__ jobs, const uint64_t* __restrict__ ptrs,
                     const void* __restrict__ items, uint32_t each, uint32_t nitems, uint32_t* counter, uint32_t kc) {
  using L = Lut<E, LEV>;
  using S = LutSmem<L::NV, W>;
  __shared__ LutShared sh;
  __shared__ LutBatchJob s_job;
  __shared__ uint2 s_item;
  const uint32_t* resident = nullptr;
  const bool one_each = nitems <= gridDim.x;
  uint32_t next = blockIdx.x;
  if (!one_each && threadIdx.x == 0) next = atomicAdd(counter, 1u);
  for (;;) {
    if (threadIdx.x == 0) {
      uint2 item = make_uint2(~0u, 0u);
      if (next < nitems)
        item = each ? make_uint2(static_cast<const uint32_t*>(items)[next / each], next % each)
                    : static_cast<const uint2*>(items)[next];
      s_item = item;
    }
    __syncthreads();
    const uint2 wi = s_item;
    if (wi.x == ~0u) break;
    if (threadIdx.x == 0) next = one_each ? nitems : atomicAdd(counter, 1u);
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
