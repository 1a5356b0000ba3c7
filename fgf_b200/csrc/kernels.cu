// kernels.cu -- sm_100a kernels of libfgfcuda.so.
//
// The byte-table kernel (Gf8, at most 4 rows and 14 sources of long rows; the
// other matrix calls run lut.cuh), the XOR of two vectors and the product of
// two vectors.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

#include "fast_core.cuh"
#include "internal.hpp"

namespace fgfc {

namespace {

// ---------------------------------------------------------------- byte-table kernel
//
// Gf8, at most 4 rows, K <= 14 sources: the RS(10,4) encode / reconstruct
// shape and the single-row ops (fast_core.cuh). Chosen per call by the tuner
// (tune.cpp): short rows use the 32-word tables (lut.cuh), which fill faster.

template <int K, bool OVR, bool SHIFT>
__global__ void __launch_bounds__(fast_threads(K, SHIFT, false), 1) matrix_fast_kernel(const __grid_constant__ MatrixLaunch a) {
  fill_fast<K>(a.tables, a.inline_tab);
  const uint32_t lane4 = (threadIdx.x & 31u) * 4u;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const uint32_t lane = threadIdx.x & 31u;
  // Head and tail, at most 8 groups: the last warp, whose columns end first. In a
  // launch of the table kernel of their own they cost 3 to 6 us a call (4 bytes
  // past 16 MiB, k = 1 10.6 -> 7.9, RS(10,4) 49.4 -> 45.3).
  const uint32_t last = gridDim.x * blockDim.x - 32u;
  if (blockIdx.x * blockDim.x + threadIdx.x >= last && lane < fast_groups(a.len, a.head, a.nvec)) {
    uint64_t off;
    const int nb = fast_group(a.len, a.head, a.nvec, lane, &off);
    fast_bytes<K>(a.src, a.dst, a.nrows, off, nb, OVR, lane4);
  }
  // SHIFT: whole warps iterate together (the row stores shuffle between lanes)
  __syncwarp();
  uint64_t vb = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x - (SHIFT ? lane : 0u);
  uint32_t wn[K][4];
  if constexpr (fast_pipe(K, SHIFT, false)) {
    const uint64_t v = SHIFT ? vb + lane : vb;
    if (vb < a.nvec) fast_load<K>(a.src, a.head + (v < a.nvec ? v : a.nvec - 1) * 16u, wn);
  }
  for (; vb < a.nvec; vb += stride) {
    const uint64_t v = SHIFT ? vb + lane : vb;
    const bool valid = !SHIFT || v < a.nvec;
    const uint64_t off = a.head + (valid ? v : a.nvec - 1) * 16u;
    uint32_t w[K][4];
    if constexpr (fast_pipe(K, SHIFT, false)) {
#pragma unroll
      for (int t = 0; t < K; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) w[t][q] = wn[t][q];
      if (vb + stride < a.nvec)
        fast_load<K>(a.src, a.head + (v + stride < a.nvec ? v + stride : a.nvec - 1) * 16u, wn);
    } else {
      if (v + stride < a.nvec) {  // this thread's next column: into L2 now
#pragma unroll
        for (int t = 0; t < K; ++t) prefetch_l2(a.src[t] + off + stride * 16u);
      }
      fast_load<K>(a.src, off, w);
    }
    uint32_t acc[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = 0;
    fast_fold<K, 4>(w, acc, lane4);
    if constexpr (SHIFT)
      store_col4_any(acc, a.dst, a.nrows, off, OVR, valid);
    else
      store_col4(acc, a.dst, a.nrows, off, OVR);
  }
}

template <int K, bool OVR, bool SHIFT>
cudaError_t launch_fast_k(const MatrixLaunch& a, cudaStream_t s) {
  cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(matrix_fast_kernel<K, OVR, SHIFT>),
                                   FastLayout<K>::smem);
  if (e != cudaSuccess) return e;
  const uint64_t want = (a.nvec + fast_threads(K, SHIFT, false) - 1) / fast_threads(K, SHIFT, false);
  const uint64_t cap = static_cast<uint64_t>(sm_count());
  const unsigned blocks = static_cast<unsigned>(want < cap ? want : cap);
  matrix_fast_kernel<K, OVR, SHIFT><<<blocks, fast_threads(K, SHIFT, false), FastLayout<K>::smem, s>>>(a);
  return cudaGetLastError();
}

template <bool OVR, bool SHIFT>
cudaError_t launch_fast_s(const MatrixLaunch& a, cudaStream_t s) {
  switch (a.k) {
    case 1: return launch_fast_k<1, OVR, SHIFT>(a, s);
    case 2: return launch_fast_k<2, OVR, SHIFT>(a, s);
    case 3: return launch_fast_k<3, OVR, SHIFT>(a, s);
    case 4: return launch_fast_k<4, OVR, SHIFT>(a, s);
    case 5: return launch_fast_k<5, OVR, SHIFT>(a, s);
    case 6: return launch_fast_k<6, OVR, SHIFT>(a, s);
    case 7: return launch_fast_k<7, OVR, SHIFT>(a, s);
    case 8: return launch_fast_k<8, OVR, SHIFT>(a, s);
    case 9: return launch_fast_k<9, OVR, SHIFT>(a, s);
    case 10: return launch_fast_k<10, OVR, SHIFT>(a, s);
    case 11: return launch_fast_k<11, OVR, SHIFT>(a, s);
    case 12: return launch_fast_k<12, OVR, SHIFT>(a, s);
    case 13: return launch_fast_k<13, OVR, SHIFT>(a, s);
    case 14: return launch_fast_k<14, OVR, SHIFT>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

template <bool OVR>
cudaError_t launch_fast(const MatrixLaunch& a, cudaStream_t s) {
  return a.shift ? launch_fast_s<OVR, true>(a, s) : launch_fast_s<OVR, false>(a, s);
}

// ---------------------------------------------------------------- helpers

__global__ void xor_kernel(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src, uint64_t len,
                           uint64_t head, uint64_t nvec) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (uint64_t v = tid; v < nvec; v += stride) {
    uint4* d = reinterpret_cast<uint4*>(dst + head + 16 * v);
    const uint4 x = ldg16(src + head + 16 * v);
    uint4 y = *d;
    y.x ^= x.x;
    y.y ^= x.y;
    y.z ^= x.z;
    y.w ^= x.w;
    *d = y;
  }
  const uint64_t tail0 = head + 16 * nvec;
  for (uint64_t i = tid; i < head + (len - tail0); i += stride) {
    const uint64_t o = i < head ? i : tail0 + (i - head);
    dst[o] ^= src[o];
  }
}

// Per-device caches (SM count) are arrays indexed by device ordinal.
constexpr int kMaxDevices = 64;

// ---- mul_elementwise where the three vectors do not share their offset
// within 16 bytes (the others run elementwise.cu).
//
// GF(2^8) products of 4 byte lanes of a 32-bit word at once by shifts and
// XORs: x * y = XOR over the set bits b of y of x * 2^b, where x * 2 is the
// byte-wise shift left reduced by the field polynomial in the lanes whose
// bit 7 falls out. A permute whose selector nibble is 8 + i copies the top
// bit of byte i over the whole byte, so each byte mask costs one PRMT.
// Gf16 and Gf32 use their tower identities over these byte products:
//   (a + b u)(c + d u) = (ac + 0x20 bd) + ((a + b)(c + d) + ac) u      (Gf16)
//   (A + B v)(C + D v) = (AC + 0x2000 BD) + ((A + B)(C + D) + AC) v   (Gf32)
// (src/field/gf16.rs:54-60, src/field/gf32.rs:36-42).

__device__ __forceinline__ uint32_t prmt_sign(uint32_t a, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(d) : "r"(a), "r"(sel));
  return d;
}

// 4 byte lanes times 2, reduced by the polynomial whose low byte is R.
template <uint32_t R>
__device__ __forceinline__ uint32_t xtime4(uint32_t x) {
  return ((x & 0x7F7F7F7Fu) << 1) ^ (prmt_sign(x, 0xBA98u) & (R * 0x01010101u));
}

// 4 independent GF(2^8) products (byte lane i of x times byte lane i of y).
template <uint32_t R>
__device__ __forceinline__ uint32_t gmul4(uint32_t x, uint32_t y) {
  uint32_t acc = 0;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    acc ^= x & prmt_sign(y << (7 - b), 0xBA98u);  // lanes whose bit b of y is set
    if (b < 7) x = xtime4<R>(x);
  }
  return acc;
}

// Two Gf16 products per word: elements [a, b] in bytes 0-1 and 2-3.
__device__ __forceinline__ uint32_t gmul16x2(uint32_t x, uint32_t y) {
  const uint32_t p = gmul4<0x1Bu>(x, y);                                   // [ac, bd, ...]
  const uint32_t q = gmul4<0x1Bu>(x ^ prmt(x, 0u, 0x2301u), y ^ prmt(y, 0u, 0x2301u));  // [(a+b)(c+d), ...]
  uint32_t c = p;                                                          // 0x20 * p: five doublings
#pragma unroll
  for (int i = 0; i < 5; ++i) c = xtime4<0x1Bu>(c);
  // [ac + 0x20 bd, (a+b)(c+d) + ac] per element
  return prmt(p, p, 0x2200u) ^ prmt(c, q, 0x7351u);
}

// The Gf16 products of two words at once (r1 = x1 * y1, r2 = x2 * y2, two
// elements each): the four cross products (a + b)(c + d) share one byte
// product pass instead of filling half of two.
__device__ __forceinline__ void gmul16x2_pair(uint32_t x1, uint32_t y1, uint32_t x2, uint32_t y2, uint32_t& r1,
                                              uint32_t& r2) {
  const uint32_t p1 = gmul4<0x1Bu>(x1, y1), p2 = gmul4<0x1Bu>(x2, y2);  // [ac, bd, ac, bd]
  const uint32_t xs = prmt(x1 ^ (x1 >> 8), x2 ^ (x2 >> 8), 0x6420u);      // a + b of the 4 elements
  const uint32_t ys = prmt(y1 ^ (y1 >> 8), y2 ^ (y2 >> 8), 0x6420u);
  const uint32_t q = gmul4<0x1Bu>(xs, ys);                                 // (a+b)(c+d) of the 4 elements
  uint32_t c = prmt(p1, p2, 0x7531u);                                      // the 4 bd, then 0x20 bd:
#pragma unroll
  for (int i = 0; i < 5; ++i) c = xtime4<0x1Bu>(c);                        // five doublings
  r1 = prmt(p1, p1, 0x2200u) ^ prmt(c, q, 0x5140u);
  r2 = prmt(p2, p2, 0x2200u) ^ prmt(c, q, 0x7362u);
}

// 0x2000 times each Gf16 lane (a + b u) of a word: 0x20 0x20 b + 0x20 (a + b) u.
// The hi lanes (a + b) take 5 doublings and the lo lanes (b) 10: the first 5
// run on both at once.
__device__ __forceinline__ uint32_t gmul2000x2(uint32_t v) {
  uint32_t w = ((v ^ (v << 8)) & 0xFF00FF00u) | ((v >> 8) & 0x00FF00FFu);
#pragma unroll
  for (int i = 0; i < 5; ++i) w = xtime4<0x1Bu>(w);
  uint32_t lo = w & 0x00FF00FFu;
#pragma unroll
  for (int i = 0; i < 5; ++i) lo = xtime4<0x1Bu>(lo);
  return (w & 0xFF00FF00u) | lo;
}

// One Gf32 product per word: [A, B] as Gf16 halves.
__device__ __forceinline__ uint32_t gmul32(uint32_t x, uint32_t y) {
  uint32_t p, q;                                                           // [AC, BD], [(A+B)(C+D), ..]
  gmul16x2_pair(x, y, x ^ prmt(x, 0u, 0x1032u), y ^ prmt(y, 0u, 0x1032u), p, q);
  const uint32_t c = gmul2000x2(p);                                        // [0x2000 AC, 0x2000 BD]
  return prmt(p ^ (c >> 16), q ^ p, 0x5410u);                             // [AC + 0x2000 BD, (A+B)(C+D) + AC]
}

// One word of 32-bit lanes holding 4 bytes of each vector (a whole number of
// elements: 4 Gf8, 2 Gf16, 1 Gf32).
template <int F>
__device__ __forceinline__ uint32_t emul_word(uint32_t x, uint32_t y) {
  if (F == kGf8B) return gmul4<0x1Bu>(x, y);
  if (F == kGf8D) return gmul4<0x1Du>(x, y);
  if (F == kGf16) return gmul16x2(x, y);
  return gmul32(x, y);
}

// One element per thread step, its bytes gathered into the low lanes of a word
// (whole elements where they are aligned): vectors that do not share their
// offset within 16 bytes, and short ones.
template <int F>
__global__ void elementwise_kernel(uint8_t* __restrict__ dst, const uint8_t* __restrict__ a,
                                   const uint8_t* __restrict__ b, uint64_t nelem) {
  constexpr int E = (F == kGf16) ? 2 : (F == kGf32 ? 4 : 1);
  const bool words = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(a) |
                       reinterpret_cast<uintptr_t>(b)) & 3u) == 0;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nelem; i += stride) {
    const uint64_t o = i * E;
    if (E == 4 && words) {
      *reinterpret_cast<uint32_t*>(dst + o) = emul_word<F>(*reinterpret_cast<const uint32_t*>(a + o),
                                                           *reinterpret_cast<const uint32_t*>(b + o));
      continue;
    }
    uint32_t x = 0, y = 0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      x |= static_cast<uint32_t>(a[o + k]) << (8 * k);
      y |= static_cast<uint32_t>(b[o + k]) << (8 * k);
    }
    const uint32_t r = emul_word<F>(x, y);
#pragma unroll
    for (int k = 0; k < E; ++k) dst[o + k] = static_cast<uint8_t>(r >> (8 * k));
  }
}

// ---- mul_elementwise over the Fan-Paar towers. Byte products use the
// byte level's log/exp tables (generator 0x2d) and a byte times the byte
// level's top generator alpha uses a 256-entry table; the 16-, 32- and 64-bit
// levels follow the Karatsuba recursion of the tower X^2 + alpha X + 1
// (src/field/fan_paar.rs:80-94, 122-134). Tables: 1 KiB, staged from
// constant memory into shared memory per CTA.
__constant__ uint8_t c_fp_tab[1024];  // exp[0..510) | pad | log[256] | alpha[256]

struct FpTab {
  const uint8_t* exp;
  const uint8_t* log;
  const uint8_t* alpha;
  __device__ __forceinline__ uint32_t m8(uint32_t a, uint32_t b) const {
    return (a && b) ? exp[log[a] + log[b]] : 0u;
  }
  __device__ __forceinline__ uint32_t alpha16(uint32_t v) const {  // v * alpha at the 16-bit level
    return (v >> 8) | (((v & 0xFFu) ^ alpha[v >> 8]) << 8);
  }
  __device__ __forceinline__ uint32_t m16(uint32_t x, uint32_t y) const {
    const uint32_t a0 = x & 0xFFu, a1 = x >> 8, b0 = y & 0xFFu, b1 = y >> 8;
    const uint32_t z0 = m8(a0, b0), z2 = m8(a1, b1), z1 = m8(a0 ^ a1, b0 ^ b1) ^ z0 ^ z2;
    return (z0 ^ z2) | ((z1 ^ alpha[z2]) << 8);
  }
  __device__ __forceinline__ uint32_t m32(uint32_t x, uint32_t y) const {
    const uint32_t a0 = x & 0xFFFFu, a1 = x >> 16, b0 = y & 0xFFFFu, b1 = y >> 16;
    const uint32_t z0 = m16(a0, b0), z2 = m16(a1, b1), z1 = m16(a0 ^ a1, b0 ^ b1) ^ z0 ^ z2;
    return (z0 ^ z2) | ((z1 ^ alpha16(z2)) << 16);
  }
  __device__ __forceinline__ uint32_t alpha32(uint32_t v) const {  // v * alpha at the 32-bit level
    return (v >> 16) | (((v & 0xFFFFu) ^ alpha16(v >> 16)) << 16);
  }
  __device__ __forceinline__ uint64_t m64(uint64_t x, uint64_t y) const {
    const uint32_t a0 = static_cast<uint32_t>(x), a1 = static_cast<uint32_t>(x >> 32);
    const uint32_t b0 = static_cast<uint32_t>(y), b1 = static_cast<uint32_t>(y >> 32);
    const uint32_t z0 = m32(a0, b0), z2 = m32(a1, b1), z1 = m32(a0 ^ a1, b0 ^ b1) ^ z0 ^ z2;
    return static_cast<uint64_t>(z0 ^ z2) | (static_cast<uint64_t>(z1 ^ alpha32(z2)) << 32);
  }
};

template <int E>
__global__ void elementwise_fp_kernel(uint8_t* __restrict__ dst, const uint8_t* __restrict__ a,
                                      const uint8_t* __restrict__ b, uint64_t nelem) {
  __shared__ uint8_t tab[1024];
  for (int i = threadIdx.x; i < 1024; i += blockDim.x) tab[i] = c_fp_tab[i];
  __syncthreads();
  const FpTab T{tab, tab + 512, tab + 768};
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nelem; i += stride) {
    uint64_t x = 0, y = 0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      x |= static_cast<uint64_t>(a[E * i + k]) << (8 * k);
      y |= static_cast<uint64_t>(b[E * i + k]) << (8 * k);
    }
    const uint64_t r = E == 1   ? T.m8(static_cast<uint32_t>(x), static_cast<uint32_t>(y))
                       : E == 2 ? T.m16(static_cast<uint32_t>(x), static_cast<uint32_t>(y))
                       : E == 4 ? T.m32(static_cast<uint32_t>(x), static_cast<uint32_t>(y))
                                : T.m64(x, y);
#pragma unroll
    for (int k = 0; k < E; ++k) dst[E * i + k] = static_cast<uint8_t>(r >> (8 * k));
  }
}

// 0x20000000 times a Gf32 element [A, B] (Gf16 halves): v = 0x2000 in the
// high half, so (A + B v) 0x2000 v = 0x2000 0x2000 B + 0x2000 (A + B) v.
__device__ __forceinline__ uint32_t gmul20000000(uint32_t w) {
  const uint32_t u = ((w ^ (w << 16)) & 0xFFFF0000u) | (w >> 16);  // [B, A + B]
  const uint32_t u1 = gmul2000x2(u);                                 // [0x2000 B, 0x2000 (A + B)]
  return (u1 & 0xFFFF0000u) | (gmul2000x2(u1) & 0x0000FFFFu);
}

__device__ __forceinline__ uint64_t ld8(const uint8_t* p) {
  if ((reinterpret_cast<uintptr_t>(p) & 7u) == 0) return *reinterpret_cast<const uint64_t*>(p);
  uint64_t v = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) v |= static_cast<uint64_t>(p[k]) << (8 * k);
  return v;
}

// GF(2^64) = Gf32[w]/(w^2 + w + 0x20000000): three word-parallel Gf32
// products and one product by the constant (src/field/gf64.rs:120-128),
// that one by doublings.
__global__ void elementwise_gf64_kernel(uint8_t* __restrict__ dst, const uint8_t* __restrict__ a,
                                        const uint8_t* __restrict__ b, uint64_t nelem) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nelem; i += stride) {
    const uint64_t x = ld8(a + 8 * i), y = ld8(b + 8 * i);
    const uint32_t p = static_cast<uint32_t>(x), q = static_cast<uint32_t>(x >> 32);
    const uint32_t c = static_cast<uint32_t>(y), d = static_cast<uint32_t>(y >> 32);
    const uint32_t ac = gmul32(p, c), bd = gmul32(q, d);
    const uint32_t lo = ac ^ gmul20000000(bd);
    const uint32_t hi = gmul32(p ^ q, c ^ d) ^ ac;
    const uint64_t r = static_cast<uint64_t>(lo) | (static_cast<uint64_t>(hi) << 32);
    uint8_t* o = dst + 8 * i;
    if ((reinterpret_cast<uintptr_t>(o) & 7u) == 0) {
      *reinterpret_cast<uint64_t*>(o) = r;
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = static_cast<uint8_t>(r >> (8 * k));
    }
  }
}

std::atomic<bool> g_fp_ready[kMaxDevices];
std::mutex g_fp_mu;

}  // namespace

int sm_count() {
  static std::atomic<int> sms[kMaxDevices];
  int dev = 0;
  cudaGetDevice(&dev);
  const bool cached = dev >= 0 && dev < kMaxDevices;
  int v = cached ? sms[dev].load(std::memory_order_relaxed) : 0;
  if (v > 0) return v;
  cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
  if (v <= 0) v = 148;
  if (cached) sms[dev].store(v, std::memory_order_relaxed);
  return v;
}

// cudaFuncSetAttribute acts on the current device only, so the opt-in to
// more than 48 KiB of dynamic shared memory is recorded per (device, kernel)
// and taken under a lock: plans, batch runners and servers may target any
// device from any host thread.
cudaError_t ensure_smem_attr(const void* fn, int bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, int> done;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(dev, fn);
  const auto it = done.find(key);
  if (it != done.end() && it->second >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done[key] = bytes;
  return e;
}

cudaError_t launch_fast_matrix(bool overwrite, const MatrixLaunch& a, cudaStream_t s) {
  return overwrite ? launch_fast<true>(a, s) : launch_fast<false>(a, s);
}

cudaError_t launch_zero_rows(uint8_t* const* rows, int n, uint64_t len, cudaStream_t s) {
  for (int j = 0; j < n; ++j) {
    cudaError_t e = cudaMemsetAsync(rows[j], 0, len, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_xor(uint8_t* dst, const uint8_t* src, uint64_t len, cudaStream_t s) {
  if (!len) return cudaSuccess;
  const uint64_t ad = reinterpret_cast<uintptr_t>(dst) & 15, as = reinterpret_cast<uintptr_t>(src) & 15;
  uint64_t head = 0, nvec = 0;
  if (ad == as) {
    head = (16 - ad) & 15;
    if (head > len) head = len;
    nvec = (len - head) / 16;
  } else {
    head = len;
  }
  const uint64_t work = nvec + head + (len - head - 16 * nvec);
  uint64_t want = (work + 255) / 256, cap = static_cast<uint64_t>(sm_count()) * 8;
  xor_kernel<<<static_cast<unsigned>(want < cap ? want : cap), 256, 0, s>>>(dst, src, len, head, nvec);
  return cudaGetLastError();
}

// Fan-Paar fields: byte tables built on the host from the tower product,
// uploaded once per device.
static cudaError_t launch_elementwise_fp(int field, uint8_t* dst, const uint8_t* a, const uint8_t* b,
                                         uint64_t len, cudaStream_t s) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  if (!g_fp_ready[dev].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lk(g_fp_mu);
    uint8_t tab[1024] = {};
    uint32_t v = 1;
    for (int i = 0; i < 255; ++i) {
      tab[i] = tab[i + 255] = static_cast<uint8_t>(v);
      tab[512 + v] = static_cast<uint8_t>(i);
      v = fp_mul(v, 0x2D, 8);
    }
    for (uint32_t x = 0; x < 256; ++x) tab[768 + x] = static_cast<uint8_t>(fp_mul_alpha(x, 8));
    e = cudaMemcpyToSymbol(c_fp_tab, tab, sizeof tab);
    if (e != cudaSuccess) return e;
    g_fp_ready[dev].store(true, std::memory_order_release);
  }
  const int E = field_bytes(field);
  const uint64_t nelem = len / E;
  uint64_t want = (nelem + 255) / 256, cap = static_cast<uint64_t>(sm_count()) * 8;
  const unsigned blocks = static_cast<unsigned>(want < cap ? want : cap);
  if (E == 1)
    elementwise_fp_kernel<1><<<blocks, 256, 0, s>>>(dst, a, b, nelem);
  else if (E == 2)
    elementwise_fp_kernel<2><<<blocks, 256, 0, s>>>(dst, a, b, nelem);
  else if (E == 4)
    elementwise_fp_kernel<4><<<blocks, 256, 0, s>>>(dst, a, b, nelem);
  else
    elementwise_fp_kernel<8><<<blocks, 256, 0, s>>>(dst, a, b, nelem);
  return cudaGetLastError();
}

// Vectors shorter than this run one element per thread: a planes warp takes
// 1 KiB times the element width through 1600 (4 bytes) to 4000 (8 bytes)
// instructions, which a short vector does not amortise. us on B200, element
// kernel / planes: Gf32 256 KiB 2.3 / 3.1, 512 KiB 3.3 / 3.3; FP32 128 KiB 3.5 /
// 3.7, 256 KiB 4.8 / 3.7; Gf64 1 MiB 7.4 / 8.9, 1.5 MiB 10.2 / 9.1; FP64 768 KiB
// 8.2 / 10.0, 1 MiB 9.9 / 10.0; Gf16 1 KiB 2.0 / 2.5, 64 KiB 2.0 / 2.45, 256 KiB
// 2.8 / 2.35. 1-byte fields (and FP16, whose log tables take 3.5) are not slower.
static uint64_t planes_min_bytes(int field) {
  switch (field) {
    case kGf16: return 1u << 17;
    case kGf32: return 1u << 19;
    case kFp32: return 1u << 18;
    case kGf64: return 5u << 18;
    case kFp64: return 1u << 20;
    default: return 0;
  }
}

cudaError_t launch_elementwise(int field, uint8_t* dst, const uint8_t* a, const uint8_t* b,
                               uint64_t len, cudaStream_t s) {
  if (!len) return cudaSuccess;
  const int E = field_bytes(field);
  if (E <= 0 || len % E) return cudaErrorInvalidValue;
  const uint64_t al = reinterpret_cast<uintptr_t>(dst) & 15, head = std::min<uint64_t>((16 - al) & 15, len);
  if (al == (reinterpret_cast<uintptr_t>(a) & 15) && al == (reinterpret_cast<uintptr_t>(b) & 15) && head % E == 0 &&
      len >= planes_min_bytes(field))
    return launch_elementwise_planes(field, dst, a, b, len, static_cast<uint32_t>(head), (len - head) / 16, s);
  if (field == kFp8 || field == kFp16 || field == kFp32 || field == kFp64)
    return launch_elementwise_fp(field, dst, a, b, len, s);
  const uint64_t nelem = len / E;
  const uint64_t want = (nelem + 255) / 256, cap = static_cast<uint64_t>(sm_count()) * 8;
  const unsigned blocks = static_cast<unsigned>(want < cap ? want : cap);
  switch (field) {
    case kGf8B: elementwise_kernel<kGf8B><<<blocks, 256, 0, s>>>(dst, a, b, nelem); break;
    case kGf8D: elementwise_kernel<kGf8D><<<blocks, 256, 0, s>>>(dst, a, b, nelem); break;
    case kGf16: elementwise_kernel<kGf16><<<blocks, 256, 0, s>>>(dst, a, b, nelem); break;
    case kGf32: elementwise_kernel<kGf32><<<blocks, 256, 0, s>>>(dst, a, b, nelem); break;
    case kGf64: elementwise_gf64_kernel<<<blocks, 256, 0, s>>>(dst, a, b, nelem); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace fgfc
