// wide.cu -- the matrix calls of the 8-byte fields where the table kernels' byte
// leaves (lut.cuh) are too much work per thread: short rows, and one or two
// sources of any length.
//
// Both fields are quadratic over a 4-byte one, so with c = c0 + c1 w and
// x = x0 + x1 w a product takes three half-products (Karatsuba) A = c0 x0,
// B = c1 x1, C = (c0 + c1)(x0 + x1), then
//   GF(2^64) (w^2 = w + beta):       lo = A + beta B, hi = A + C
//   Fan-Paar (X^2 = alpha X + 1):    lo = A + B,      hi = A + C + (1 + alpha) B
// on the sums over all sources. A half-product is 8 lookups in 16-word tables,
// conflict-free as the table kernels' (lanes at different words are at different
// banks); the fix-up takes 8 more per row. A thread has one element, half of a
// table kernel's column, up to 8 rows in one launch, and no more code than one
// source's, so where a thread gets one column anyway (short rows) or the fix-up
// outweighs the lookups (few sources) it ends first. Latency bounds the former, the
// lookups the latter. us on B200, table kernels -> this one, GF(2^64): 64 KiB of
// k = 4, m = 3 11.6 -> 7.8, m = 6 21.9 -> 10.4; 300000 bytes at odd addresses,
// k = 10, m = 4 28.7 -> 14.6; 16 MiB of k = 1, m = 4 59.1 -> 42.1.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "lut.cuh"

namespace fgfc {

namespace {

constexpr int kWideRows = 8;                    // rows per launch
constexpr int kWideThreads = 256;
constexpr size_t kWideSmemMax = 160 * 1024;     // tables of one CTA
constexpr uint32_t kWideTables = 12;            // tables of a coefficient: (A, B, C) x 4 input bytes
constexpr uint32_t kTableWords = 32;            // low nibble's 16 words, high nibble's 16

// Resident CTAs; 16 MiB of eight rows added, k = 1, with 2, 3, 4, 5: 163, 122, 107, 96 us.
constexpr int wide_ctas(size_t rows) { return rows <= 4 ? 6 : 5; }

struct WideLaunch {
  const uint32_t* img;  // images of coefficient (t, j) at ((t0 + t) * cols + r0 + j) * kWideTables * 8
  uint32_t cols, k, ovr;
  uint64_t nelem;
  const uint8_t* src[kMaxSrc];
  uint8_t* dst[kWideRows];
};

__device__ __forceinline__ uint64_t load8(const uint8_t* p) {
  if ((reinterpret_cast<uintptr_t>(p) & 7u) == 0) return *reinterpret_cast<const uint64_t*>(p);
  uint64_t v = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) v |= static_cast<uint64_t>(p[i]) << (8 * i);
  return v;
}

__device__ __forceinline__ void store8(uint8_t* p, uint64_t v, bool ovr) {
  if ((reinterpret_cast<uintptr_t>(p) & 7u) == 0) {
    uint64_t* q = reinterpret_cast<uint64_t*>(p);
    *q = ovr ? v : (*q ^ v);
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint8_t b = static_cast<uint8_t>(v >> (8 * i));
    p[i] = ovr ? b : static_cast<uint8_t>(p[i] ^ b);
  }
}

// acc[j] ^= the M maps of x whose tables start at byte `base`, input byte p's at
// base + p * M * 128.
template <int M>
__device__ __forceinline__ void fold_half(uint32_t (&acc)[M], uint32_t base, uint32_t x) {
  const uint32_t lo = x & 0x0F0F0F0Fu, hi = (x >> 2) & 0x3C3C3C3Cu;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const uint32_t a = lut_addr<4>(lo, base, p), b = lut_addr<1>(hi, base, p);
#pragma unroll
    for (int j = 0; j < M; ++j) {
      const uint32_t o = (p * M + j) * 4u * kTableWords;
      acc[j] ^= lds_at(a + o) ^ lds_at(b + o + 64u);
    }
  }
}

template <int M, bool FP>
__global__ void __launch_bounds__(kWideThreads, wide_ctas(M)) wide_kernel(const __grid_constant__ WideLaunch a) {
  constexpr uint32_t kSource = kWideTables * M * kTableWords;  // words of one source's tables
  uint32_t* tab = reinterpret_cast<uint32_t*>(g_smem);
  for (uint32_t i = threadIdx.x; i < a.k * kSource; i += blockDim.x) {
    const uint32_t slot = i / kTableWords, j = slot % M, s = slot / M % kWideTables, t = slot / (M * kWideTables);
    const uint32_t* im = a.img + ((static_cast<size_t>(t) * a.cols + j) * kWideTables + s) * 8 + (i >> 4 & 1u) * 4;
    const uint4 v = *reinterpret_cast<const uint4*>(im);
    tab[i] = (v.x & (0u - (i & 1u))) ^ (v.y & (0u - (i >> 1 & 1u))) ^ (v.z & (0u - (i >> 2 & 1u))) ^
             (v.w & (0u - (i >> 3 & 1u)));
  }
  const uint32_t fix = a.k * kSource * 4u;
  for (uint32_t i = threadIdx.x; i < 4 * kTableWords; i += blockDim.x) {
    const uint32_t v = (i & 15u) << (8 * (i / kTableWords) + (i >> 4 & 1u) * 4);
    tab[fix / 4 + i] = FP ? v ^ lut_const1<4, true>(v) : lut_const1<4, false>(v);
  }
  __syncthreads();
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t e = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < a.nelem; e += stride) {
    uint32_t accA[M], accB[M], accC[M];
#pragma unroll
    for (int j = 0; j < M; ++j) accA[j] = accB[j] = accC[j] = 0;
    uint64_t next = load8(a.src[0] + 8 * e);
    uint32_t base = 0;
    for (uint32_t t = 0; t < a.k; ++t) {
      const uint64_t x = next;  // the next source's element is in flight during this one's lookups
      if (t + 1 < a.k) next = load8(a.src[t + 1] + 8 * e);
      const uint32_t x0 = static_cast<uint32_t>(x), x1 = static_cast<uint32_t>(x >> 32);
      fold_half<M>(accA, base, x0);
      fold_half<M>(accB, base + kSource * 4u / 3u, x1);
      fold_half<M>(accC, base + kSource * 8u / 3u, x0 ^ x1);
      base += kSource * 4u;
    }
#pragma unroll
    for (int j = 0; j < M; ++j) {
      uint32_t f[1] = {0};
      fold_half<1>(f, fix, accB[j]);
      const uint32_t lo = accA[j] ^ (FP ? accB[j] : f[0]), hi = accA[j] ^ accC[j] ^ (FP ? f[0] : 0u);
      store8(a.dst[j] + 8 * e, static_cast<uint64_t>(lo) | (static_cast<uint64_t>(hi) << 32), a.ovr != 0);
    }
  }
}

template <bool FP>
const void* wide_kernel_for(size_t rows) {
  switch (rows) {
    case 1: return reinterpret_cast<const void*>(wide_kernel<1, FP>);
    case 2: return reinterpret_cast<const void*>(wide_kernel<2, FP>);
    case 3: return reinterpret_cast<const void*>(wide_kernel<3, FP>);
    case 4: return reinterpret_cast<const void*>(wide_kernel<4, FP>);
    case 5: return reinterpret_cast<const void*>(wide_kernel<5, FP>);
    case 6: return reinterpret_cast<const void*>(wide_kernel<6, FP>);
    case 7: return reinterpret_cast<const void*>(wide_kernel<7, FP>);
    default: return reinterpret_cast<const void*>(wide_kernel<8, FP>);
  }
}

}  // namespace

// Where the lines lie (table kernels / this one, us): GF(2^64) RS(10,4) 256 KiB 20.1 /
// 14.5, 512 KiB 15.2 / 18.2; k = 10, m = 6 (two launches there) 512 KiB 27.9 / 29.2,
// k = 3, m = 6 13.5 / 11.0, 1 MiB 15.1 / 16.8; k = 1, m = 1 512 KiB 3.4 / 3.2, 1 MiB
// 3.8 / 3.7; 16 MiB of k = 1, m = 2 34.7 / 24.0, k = 2, m = 2 41.9 / 38.8, FP64 24.3
// / 24.3 and 32.7 / 38.6, k = 1, m = 3 46.9 / 32.7, k = 2, m = 3 60.4 / 53.9, m = 4
// 61.7 / 70.3, m = 8 added 163 / 139.
bool wide_chosen(int field, size_t k, size_t m, size_t len) {
  if (field_bytes(field) != 8) return false;
  if (len < (k <= 2 || m > 4 ? 768u << 10 : 512u << 10)) return true;
  if (field == kFp64) return (k == 1 && m >= 3) || (k == 2 && (m == 3 || m > 4));
  return k <= 2 && m >= 2;
}

// Long stripes of few sources gain more from this kernel than from sharing the
// GPU. Table kernels' work list / a launch each, us: two of 8 MiB GF(2^64) k = 1, m
// = 3 65 / 40, k = 2, m = 2 53 / 45, FP64 k = 1, m = 4 55 / 50, k = 2, m = 8 123 / 140;
// four of 4 MiB GF(2^64) k = 1, m = 2 41 / 41, m = 3 65 / 50, k = 2, m = 4 82 / 94, FP64
// k = 1, m = 4 55 / 60.
bool wide_stripe(int field, size_t k, size_t m, size_t len) {
  if (len < (4u << 20) || !wide_chosen(field, k, m, len)) return false;
  return len >= (8u << 20) ? !(field == kFp64 && k == 2 && m > 4) : field == kGf64 && k == 1;
}

cudaError_t wide_launch(int field, const uint8_t* const* srcs, size_t k, uint8_t* const* rows, size_t m,
                        const uint32_t* img, size_t len, bool overwrite, cudaStream_t stream) {
  const uint64_t nelem = len / 8;
  WideLaunch a;
  a.cols = static_cast<uint32_t>(m);
  a.nelem = nelem;
  for (size_t r0 = 0; r0 < m; r0 += kWideRows) {
    const size_t nr = std::min<size_t>(kWideRows, m - r0);
    const size_t per_src = kWideTables * nr * kTableWords * 4, fix = 4 * kTableWords * 4;
    const size_t kc = std::min<size_t>(kMaxSrc, (kWideSmemMax - fix) / per_src);
    const void* fn = field == kFp64 ? wide_kernel_for<true>(nr) : wide_kernel_for<false>(nr);
    cudaError_t e = ensure_smem_attr(fn, static_cast<int>(kWideSmemMax));
    if (e != cudaSuccess) return e;
    for (size_t j = 0; j < nr; ++j) a.dst[j] = rows[r0 + j];
    for (size_t t0 = 0; t0 < k; t0 += kc) {
      const size_t kk = std::min(kc, k - t0);
      a.img = img + (t0 * m + r0) * kWideTables * 8;
      a.k = static_cast<uint32_t>(kk);
      a.ovr = overwrite && t0 == 0 ? 1u : 0u;
      for (size_t t = 0; t < kk; ++t) a.src[t] = srcs[t0 + t];
      const size_t smem = kk * per_src + fix;
      const uint64_t want = (nelem + kWideThreads - 1) / kWideThreads;
      const uint64_t per_sm = std::max<uint64_t>(1, std::min<uint64_t>(wide_ctas(nr), (220 * 1024) / smem));
      const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(want, static_cast<uint64_t>(sm_count()) * per_sm));
      void* args[] = {&a};
      e = cudaLaunchKernel(fn, dim3(grid), dim3(kWideThreads), args, smem, stream);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace fgfc
