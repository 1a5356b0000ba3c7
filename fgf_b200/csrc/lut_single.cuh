// lut_single.cuh -- one call's table kernel (lut.cuh): grid-stride over the
// tiles of one job, tables filled once per CTA. Instantiated per element
// width in lut_e1.cu, lut_e2.cu, lut_e4.cu and lut_e8.cu.
#pragma once
#include "lut.cuh"

namespace fgfc {

// CTAs per SM the register budget is set for: accumulators (3^LEV leaf
// products x W words x 16 / E elements) plus three sources and their packed words.
template <int E, int LEV, int W, bool UNAL>
constexpr int lut_min_ctas() {
  return pow3(LEV) * W * (16 / E) <= 16 ? (UNAL ? 3 : 4) : pow3(LEV) * W * (16 / E) <= 32 && !UNAL ? 3 : 2;
}

template <int E, int LEV, int W, bool UNAL>
__global__ void __launch_bounds__(kLutThreads, lut_min_ctas<E, LEV, W, UNAL>())
    lut_kernel(const __grid_constant__ LutArgs a) {
  using L = Lut<E, LEV>;
  using S = LutSmem<L::NV, W>;
  __shared__ LutShared sh;
  for (uint32_t i = threadIdx.x; i < a.g.k; i += blockDim.x) sh.src[i] = a.src[i];
  for (uint32_t i = threadIdx.x; i < a.g.nrows; i += blockDim.x) sh.dst[i] = a.dst[i];
  lut_fill<L, W>(a.img ? a.img : a.inl, a.g.k);
  __syncthreads();
  const bool ovr = a.g.ovr != 0, fp = a.fp != 0;
  const uint32_t nwork = gridDim.x - a.edge_cta;
  if (blockIdx.x == nwork) {
    uint8_t* stage = g_smem + a.g.k / 3u * S::block3 + a.g.k % 3u * S::block1;
    lut_edges<L, LEV, W, UNAL>(a.g, sh, stage, ovr, fp);
    return;
  }
  if (a.ntiles) lut_run<L, LEV, W, UNAL>(a.g, sh, blockIdx.x, nwork, ovr, fp);
}

// Launch one job of this (LEV, W); `a` is complete but for its tiling.
template <int E, int LEV, int W, bool UNAL>
cudaError_t lut_launch_one(LutArgs& a, cudaStream_t s, bool edges_only) {
  using L = Lut<E, LEV>;
  using S = LutSmem<L::NV, W>;
  auto kern = lut_kernel<E, LEV, W, UNAL>;
  const bool edges = lut_has_edges(a.g, UNAL);
  const size_t smem = a.g.k / 3 * S::block3 + a.g.k % 3 * S::block1 + (edges ? a.g.k * kEdges * 16 : 0);
  cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(kern), kLutSmemMax);
  if (e != cudaSuccess) return e;
  const uint64_t sms = static_cast<uint64_t>(sm_count());
  // Small calls take narrower CTAs, so that every SM gets one.
  unsigned threads = kLutThreads;
  const uint64_t cols = edges_only ? 0 : UNAL && !a.g.bytes ? lut_unal_blocks(a.g.ncol) * 32 / kUnalStep : a.g.len / 16;
  while (threads > 64 && cols < sms * threads) threads /= 2;
  a.edge_cta = edges ? 1u : 0u;
  a.ntiles = edges_only ? 0 : lut_tiles(a.g, UNAL, threads);
  const uint64_t cap = sms * lut_min_ctas<E, LEV, W, UNAL>();
  const unsigned grid = static_cast<unsigned>(a.ntiles < cap ? a.ntiles : cap) + a.edge_cta;
  if (!grid) return cudaSuccess;
  kern<<<grid, threads, smem, s>>>(a);
  return cudaGetLastError();
}

template <int E, int LEV, int W>
cudaError_t lut_launch_lw(LutArgs& a, cudaStream_t s, bool unal, bool edges_only) {
  return unal ? lut_launch_one<E, LEV, W, true>(a, s, edges_only) : lut_launch_one<E, LEV, W, false>(a, s, edges_only);
}

}  // namespace fgfc
