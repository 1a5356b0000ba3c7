// lut_single.cuh -- one call's table kernel (lut.cuh): grid-stride over the
// tiles of one job, tables filled once per CTA. Instantiated per element
// width in lut_e1.cu, lut_e2.cu, lut_e4.cu and lut_e8.cu.
#pragma once
#include "lut.cuh"

namespace fgfc {

// CTAs per SM the register budget is set for: accumulators (3^LEV leaf products
// x W words x 16 / E elements) plus two sets of three sources and their packed
// words. Fewer, larger budgets win over more CTAs once the next column is
// fetched ahead (16 accumulators, 4 -> 3 CTAs and ahead: Gf8D RS(10,4) 4 MiB
// 17.6 -> 16.2 us; 4 and 6 accumulators, 4 -> 3: Gf32 RS(10,1) 4 MiB 16.4 -> 15.7,
// GF(2^64) RS(8,1) 20.4 -> 19.7), but for the 2-byte rows without a split
// (RS(10,2) 8 MiB 27.0 against 28.9); unaligned rows of 24 and 32 spill at 3.
template <int E, int LEV, int W, int MODE>
constexpr int lut_min_ctas() {
  constexpr int n = pow3(LEV) * W * (16 / E);
  return E == 2 && LEV == 0 && W == 1 && MODE != kAnyOff ? 4 : n <= 16 ? 3 : n <= 32 && MODE == kAligned ? 3 : 2;
}

template <int E, int LEV, int W, int MODE>
__global__ void __launch_bounds__(kLutThreads, lut_min_ctas<E, LEV, W, MODE>())
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
    lut_edges<L, LEV, W, MODE>(a.g, sh, stage, ovr, fp);
    return;
  }
  lut_run<L, LEV, W, MODE>(a.g, sh, blockIdx.x, nwork, ovr, fp);
}

// Launch one job of this (LEV, W); `a` is complete but for its tiling.
template <int E, int LEV, int W, int MODE>
cudaError_t lut_launch_one(LutArgs& a, cudaStream_t s) {
  using L = Lut<E, LEV>;
  using S = LutSmem<L::NV, W>;
  auto kern = lut_kernel<E, LEV, W, MODE>;
  const bool edges = lut_has_edges(a.g, MODE);
  const size_t smem = a.g.k / 3 * S::block3 + a.g.k % 3 * S::block1 + (edges ? (a.g.k + kLutRows) * kEdges * 16 : 0);
  cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(kern), kLutSmemMax);
  if (e != cudaSuccess) return e;
  const uint64_t sms = static_cast<uint64_t>(sm_count());
  // Small calls take narrower CTAs, so that every SM gets one.
  unsigned threads = kLutThreads;
  const uint64_t cols = a.g.len / 16;
  while (threads > 64 && cols < sms * threads) threads /= 2;
  a.edge_cta = edges ? 1u : 0u;
  a.ntiles = lut_tiles(a.g, MODE, threads);
  const uint64_t cap = sms * lut_min_ctas<E, LEV, W, MODE>();
  const unsigned grid = static_cast<unsigned>(a.ntiles < cap ? a.ntiles : cap) + a.edge_cta;
  if (!grid) return cudaSuccess;
  kern<<<grid, threads, smem, s>>>(a);
  return cudaGetLastError();
}

template <int E, int LEV, int W>
cudaError_t lut_launch_lw(LutArgs& a, cudaStream_t s, int mode) {
  return mode == kAligned   ? lut_launch_one<E, LEV, W, kAligned>(a, s)
         : mode == kRowsOff ? lut_launch_one<E, LEV, W, kRowsOff>(a, s)
                            : lut_launch_one<E, LEV, W, kAnyOff>(a, s);
}

}  // namespace fgfc
