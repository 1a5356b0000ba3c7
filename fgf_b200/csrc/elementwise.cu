// elementwise.cu -- the product of two vectors, bit-sliced.
//
// A thread takes 32 elements of both vectors, transposes them into bit planes
// (one 32-bit word per bit of the element, one bit per element) and multiplies
// plane by plane: one LOP3 (and, xor) per pair of input bits, the tower levels
// by Karatsuba, reductions and tower constants as XORs of planes. Both inputs
// are data here, so no table helps; shift-and-mask products of packed bytes
// cost 9 to 85 operations per byte (1- to 8-byte elements), the planes cost 5
// to 16, transposes included. 1-byte fields run at HBM's rate, the others are
// bound by the ALU pipe (HBM's time is worth about 8 operations per byte). us on B200, 64 MiB
// vectors, shift-and-mask (Fan-Paar: log tables) -> planes:
//   Gf8D 44.6 -> 32.7   Gf16 77.2 -> 40.4   Gf32 185 -> 54   Gf64 322 -> 85
//   FP8  149 -> 35      FP16 129 -> 44      FP32 168 -> 66   FP64 246 -> 97
// (FP64 holds more planes than registers: 256 bytes a thread go through local memory.)
//
// The order of elements within a transposed block does not matter as long as
// all three vectors use the same, so a thread's words are whichever 16-byte
// vectors coalesce: vector j of lane l is base + 32 j + l.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "fast_core.cuh"
#include "internal.hpp"

namespace fgfc {

namespace {

// ---------------------------------------------------------------- three-input logic

// Written out: left to itself the compiler rebalances the XOR chains and spends
// a quarter more instructions on them (ALU instructions per 32 products: 245 ->
// 172 for 1 byte, 661 -> 504 for Gf16, 1911 -> 1554 for Gf32; 64 MiB of Gf16
// 47.8 -> 40.6 us).
template <uint32_t LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
  return d;
}
__device__ __forceinline__ uint32_t and_xor(uint32_t a, uint32_t b, uint32_t c) { return lop3<0x6Au>(a, b, c); }
__device__ __forceinline__ uint32_t xor3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0x96u>(a, b, c); }
// m ? a : b, bit by bit
__device__ __forceinline__ uint32_t pick(uint32_t m, uint32_t a, uint32_t b) { return lop3<0xCAu>(m, a, b); }

// ---------------------------------------------------------------- bit planes

// Right shifts of the transposes on the multiply pipe: 64 MiB products of 1-
// and 2-byte elements 42.9 -> 41.6 and 54.5 -> 50.5 us; wider ones lose.
template <int E>
constexpr bool kMulShift = E <= 2;

// 8x8 bit transpose in each byte lane of 8 words (its own inverse).
template <bool MUL>
__device__ __forceinline__ void swap_bits(uint32_t& a, uint32_t& b, int s, uint32_t m, const Shift<MUL>& sh) {
  const uint32_t x = pick(m, a, b << s);
  b = pick(m, sh.shr(a, s), b);
  a = x;
}
template <bool MUL>
__device__ __forceinline__ void planes8(uint32_t* w, const Shift<MUL>& sh) {
#pragma unroll
  for (int i = 0; i < 4; ++i) swap_bits(w[i], w[i + 4], 4, 0x0F0F0F0Fu, sh);
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (!(i & 2)) swap_bits(w[i], w[i + 2], 2, 0x33333333u, sh);
#pragma unroll
  for (int i = 0; i < 8; i += 2) swap_bits(w[i], w[i + 1], 1, 0x55555555u, sh);
}

// 2 E vectors of 16 bytes to 8 E planes, plane 8 p + b for bit b of byte p.
template <int E>
__device__ __forceinline__ void to_planes(const uint4 (&x)[2 * E], uint32_t (&a)[8 * E], const Shift<kMulShift<E>>& sh) {
#pragma unroll
  for (int v = 0; v < 2 * E; ++v) {
    if constexpr (E == 1) {
      a[4 * v] = x[v].x, a[4 * v + 1] = x[v].y, a[4 * v + 2] = x[v].z, a[4 * v + 3] = x[v].w;
    } else if constexpr (E == 2) {
      a[2 * v] = prmt(x[v].x, x[v].y, 0x6420u), a[8 + 2 * v] = prmt(x[v].x, x[v].y, 0x7531u);
      a[2 * v + 1] = prmt(x[v].z, x[v].w, 0x6420u), a[8 + 2 * v + 1] = prmt(x[v].z, x[v].w, 0x7531u);
    } else if constexpr (E == 4) {
      const uint32_t p = prmt(x[v].x, x[v].y, 0x5140u), q = prmt(x[v].z, x[v].w, 0x5140u);
      const uint32_t r = prmt(x[v].x, x[v].y, 0x7362u), s = prmt(x[v].z, x[v].w, 0x7362u);
      a[v] = prmt(p, q, 0x5410u), a[8 + v] = prmt(p, q, 0x7632u);
      a[16 + v] = prmt(r, s, 0x5410u), a[24 + v] = prmt(r, s, 0x7632u);
    } else if (v % 2 == 0) {  // two vectors: 4 elements
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t w0 = h ? x[v].y : x[v].x, w1 = h ? x[v].w : x[v].z;
        const uint32_t w2 = h ? x[v + 1].y : x[v + 1].x, w3 = h ? x[v + 1].w : x[v + 1].z;
        const uint32_t p = prmt(w0, w1, 0x5140u), q = prmt(w2, w3, 0x5140u);
        const uint32_t r = prmt(w0, w1, 0x7362u), s = prmt(w2, w3, 0x7362u);
        a[32 * h + v / 2] = prmt(p, q, 0x5410u), a[32 * h + 8 + v / 2] = prmt(p, q, 0x7632u);
        a[32 * h + 16 + v / 2] = prmt(r, s, 0x5410u), a[32 * h + 24 + v / 2] = prmt(r, s, 0x7632u);
      }
    }
  }
#pragma unroll
  for (int p = 0; p < E; ++p) planes8(a + 8 * p, sh);
}

// The inverse; `a` is clobbered.
template <int E>
__device__ __forceinline__ void from_planes(uint32_t (&a)[8 * E], uint4 (&x)[2 * E], const Shift<kMulShift<E>>& sh) {
#pragma unroll
  for (int p = 0; p < E; ++p) planes8(a + 8 * p, sh);
#pragma unroll
  for (int v = 0; v < 2 * E; ++v) {
    if constexpr (E == 1) {
      x[v] = make_uint4(a[4 * v], a[4 * v + 1], a[4 * v + 2], a[4 * v + 3]);
    } else if constexpr (E == 2) {
      x[v].x = prmt(a[2 * v], a[8 + 2 * v], 0x5140u), x[v].y = prmt(a[2 * v], a[8 + 2 * v], 0x7362u);
      x[v].z = prmt(a[2 * v + 1], a[8 + 2 * v + 1], 0x5140u), x[v].w = prmt(a[2 * v + 1], a[8 + 2 * v + 1], 0x7362u);
    } else if constexpr (E == 4) {
      const uint32_t p = prmt(a[v], a[8 + v], 0x5140u), q = prmt(a[16 + v], a[24 + v], 0x5140u);
      const uint32_t r = prmt(a[v], a[8 + v], 0x7362u), s = prmt(a[16 + v], a[24 + v], 0x7362u);
      x[v] = make_uint4(prmt(p, q, 0x5410u), prmt(p, q, 0x7632u), prmt(r, s, 0x5410u), prmt(r, s, 0x7632u));
    } else if (v % 2 == 0) {
      uint32_t w[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t* b = a + 32 * h + v / 2;
        const uint32_t p = prmt(b[0], b[8], 0x5140u), q = prmt(b[16], b[24], 0x5140u);
        const uint32_t r = prmt(b[0], b[8], 0x7362u), s = prmt(b[16], b[24], 0x7362u);
        w[h][0] = prmt(p, q, 0x5410u), w[h][1] = prmt(p, q, 0x7632u);
        w[h][2] = prmt(r, s, 0x5410u), w[h][3] = prmt(r, s, 0x7632u);
      }
      x[v] = make_uint4(w[0][0], w[1][0], w[0][1], w[1][1]);
      x[v + 1] = make_uint4(w[0][2], w[1][2], w[0][3], w[1][3]);
    }
  }
}

// ---------------------------------------------------------------- products of planes

enum Family { kPoly1B, kPoly1D, kFanPaar };  // flat bytes mod 0x11B (and its towers), mod 0x11D, Fan-Paar

// beta of the towers over 0x11B: 0x20 = x^5 for bytes (x^8 .. x^12 reduced),
// one level up beta (b0, b1) = (beta beta b1, beta (b0 + b1)).
template <int N>
__device__ __forceinline__ void mul_beta(const uint32_t* v, uint32_t* o) {
  if constexpr (N == 8) {
    const uint32_t a = v[3] ^ v[7], b = v[4] ^ v[5];
    o[0] = a;
    o[1] = a ^ v[4];
    o[2] = b;
    o[3] = xor3(a, v[5], v[6]);
    o[4] = xor3(v[3], v[4], v[6]);
    o[5] = xor3(b, v[0], v[7]);
    o[6] = xor3(v[1], v[5], v[6]);
    o[7] = xor3(v[2], v[6], v[7]);
  } else {
    constexpr int M = N / 2;
    uint32_t s[M], t[M];
    mul_beta<M>(v + M, t);
    mul_beta<M>(t, o);
#pragma unroll
    for (int i = 0; i < M; ++i) s[i] = v[i] ^ v[M + i];
    mul_beta<M>(s, o + M);
  }
}

// alpha of the Fan-Paar level of N bits: (a0, a1) -> (a1, a0 + alpha' a1).
template <int N>
__device__ __forceinline__ void mul_alpha(const uint32_t* v, uint32_t* o) {
  if constexpr (N == 1) {
    o[0] = v[0];
  } else {
    constexpr int M = N / 2;
    uint32_t t[M];
    mul_alpha<M>(v + M, t);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      o[i] = v[M + i];
      o[M + i] = v[i] ^ t[i];
    }
  }
}

// c = a b over the field of N bits.
template <int N, Family F>
__device__ __forceinline__ void mul_planes(const uint32_t* a, const uint32_t* b, uint32_t* c) {
  if constexpr (F != kFanPaar && N == 8) {
    uint32_t p[15];
#pragma unroll
    for (int k = 0; k < 15; ++k) {
      const int lo = k < 8 ? 0 : k - 7, hi = k < 8 ? k : 7;
      p[k] = a[lo] & b[k - lo];
#pragma unroll
      for (int i = lo + 1; i <= hi; ++i) p[k] = and_xor(a[i], b[k - i], p[k]);
    }
    // x^8 .. x^14 reduced, for each power of the result the ones that reach it
    if constexpr (F == kPoly1D) {  // x^8 = x^4 + x^3 + x^2 + 1
      c[0] = xor3(xor3(p[0], p[8], p[12]), p[13], p[14]);
      c[1] = xor3(p[1], p[9], p[13]) ^ p[14];
      c[2] = xor3(xor3(p[2], p[8], p[10]), p[12], p[13]);
      c[3] = xor3(xor3(p[3], p[8], p[9]), p[11], p[12]);
      c[4] = xor3(xor3(p[4], p[8], p[9]), p[10], p[14]);
      c[5] = xor3(p[5], p[9], p[10]) ^ p[11];
      c[6] = xor3(p[6], p[10], p[11]) ^ p[12];
      c[7] = xor3(p[7], p[11], p[12]) ^ p[13];
    } else {  // x^8 = x^4 + x^3 + x + 1
      c[0] = xor3(p[0], p[8], p[12]) ^ p[13];
      c[1] = xor3(xor3(p[1], p[8], p[9]), p[12], p[14]);
      c[2] = xor3(p[2], p[9], p[10]) ^ p[13];
      c[3] = xor3(xor3(xor3(p[3], p[8], p[10]), p[11], p[12]), p[13], p[14]);
      c[4] = xor3(xor3(p[4], p[8], p[9]), p[11], p[14]);
      c[5] = xor3(p[5], p[9], p[10]) ^ p[12];
      c[6] = xor3(p[6], p[10], p[11]) ^ p[13];
      c[7] = xor3(p[7], p[11], p[12]) ^ p[14];
    }
  } else if constexpr (F == kFanPaar && N == 2) {
    c[0] = and_xor(a[1], b[1], a[0] & b[0]);
    c[1] = and_xor(a[1], b[0] ^ b[1], a[0] & b[1]);
  } else {
    constexpr int M = N / 2;
    uint32_t z0[M], z2[M], t[M], sa[M], sb[M];
    mul_planes<M, F>(a, b, z0);
    mul_planes<M, F>(a + M, b + M, z2);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      sa[i] = a[i] ^ a[M + i];
      sb[i] = b[i] ^ b[M + i];
    }
    mul_planes<M, F>(sa, sb, c + M);
    if constexpr (F == kFanPaar)
      mul_alpha<M>(z2, t);
    else
      mul_beta<M>(z2, t);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      c[i] = z0[i] ^ (F == kFanPaar ? z2[i] : t[i]);
      c[M + i] = F == kFanPaar ? xor3(c[M + i] ^ z0[i], z2[i], t[i]) : c[M + i] ^ z0[i];
    }
  }
}

// ---------------------------------------------------------------- kernel

// An element at p, bytewise, in the low bytes of a vector.
template <int E>
__device__ __forceinline__ uint4 get_element(const uint8_t* p) {
  uint32_t w[2] = {0, 0};
#pragma unroll
  for (int i = 0; i < E; ++i) w[i / 4] |= static_cast<uint32_t>(p[i]) << (8 * (i & 3));
  return make_uint4(w[0], w[1], 0, 0);
}
template <int E>
__device__ __forceinline__ void put_element(uint8_t* p, const uint4& v) {
#pragma unroll
  for (int i = 0; i < E; ++i) p[i] = static_cast<uint8_t>((i < 4 ? v.x : v.y) >> (8 * (i & 3)));
}

// nvec 16-byte vectors from byte `head` on, whole warps taking blocks of 64 E;
// the last block ends where the vectors do. One more block is the head and the
// tail, fewer than 16 bytes each: an element of the head per lane, one of the
// tail per lane from lane 16 on. It goes through the same code: a second copy of
// the product for the edges alone took longer to fetch than to run (8 bytes past
// a boundary, us, copy -> same code: Gf8D 64 KiB 2.9 -> 2.0, FP64 1.5 MiB 15.5 ->
// 10.4, Gf64 64 MiB 90 -> 85). The next block's vectors are in flight during the
// product where registers allow it.
template <int E, Family F>
__global__ void __launch_bounds__(128) elementwise_planes_kernel(uint8_t* dst, const uint8_t* a, const uint8_t* b,
                                                                 uint64_t len, uint32_t head, uint64_t nvec) {
  constexpr int V = 2 * E;
  constexpr bool kAhead = E <= 2;
  const Shift<kMulShift<E>> sh;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t nblocks = (nvec + 32 * V - 1) / (32 * V);
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (blockDim.x / 32);
  const uint64_t tail0 = head + 16 * nvec;
  const uint64_t total = nblocks + (head || tail0 != len ? 1 : 0);
  // this lane's element of the edge block
  const uint64_t eo = (lane < 16 ? 0 : tail0) + (lane & 15u) * E;
  const bool edge = eo < (lane < 16 ? head : len);
  uint64_t blk = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32;
  uint4 x[V], y[V];
  uint32_t pa[8 * E], pb[8 * E], pc[8 * E];
  // whole blocks (all but the last one) go by one base address per vector
  const uint64_t whole = nvec / (32 * V);
  const auto load = [&](uint64_t q) {
    const uint64_t o = head + 16 * (q * (32 * V) + lane);
    if (q < whole) {
#pragma unroll
      for (int j = 0; j < V; ++j) {
        x[j] = ldg16(a + o + 512 * j);
        y[j] = ldg16(b + o + 512 * j);
      }
    } else {
      const uint32_t left = q < nblocks ? static_cast<uint32_t>(nvec - q * (32 * V)) : 0u;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        x[j] = y[j] = make_uint4(0, 0, 0, 0);
        if (32 * j + lane < left) {
          x[j] = ldg16(a + o + 512 * j);
          y[j] = ldg16(b + o + 512 * j);
        }
      }
      if (q == nblocks && edge) {
        x[0] = get_element<E>(a + eo);
        y[0] = get_element<E>(b + eo);
      }
    }
  };
  if (kAhead && blk < total) load(blk);
  for (; blk < total; blk += warps) {
    if (!kAhead) load(blk);
    to_planes<E>(x, pa, sh);
    to_planes<E>(y, pb, sh);
    if (kAhead && blk + warps < total) load(blk + warps);
    mul_planes<8 * E, F>(pa, pb, pc);
    uint4 r[V];
    from_planes<E>(pc, r, sh);
    uint8_t* o = dst + head + 16 * (blk * (32 * V) + lane);
    if (blk < whole) {
#pragma unroll
      for (int j = 0; j < V; ++j) *reinterpret_cast<uint4*>(o + 512 * j) = r[j];
    } else {
      const uint32_t left = blk < nblocks ? static_cast<uint32_t>(nvec - blk * (32 * V)) : 0u;
#pragma unroll
      for (int j = 0; j < V; ++j)
        if (32 * j + lane < left) *reinterpret_cast<uint4*>(o + 512 * j) = r[j];
      if (blk == nblocks && edge) put_element<E>(dst + eo, r[0]);
    }
  }
}

template <int E, Family F>
cudaError_t launch(uint8_t* dst, const uint8_t* a, const uint8_t* b, uint64_t len, uint32_t head, uint64_t nvec,
                   cudaStream_t s) {
  const uint64_t nblocks = (nvec + 64 * E - 1) / (64 * E) + 1;  // and the edges
  const uint64_t sms = static_cast<uint64_t>(sm_count());
  // Short vectors take one-warp CTAs, so that every SM gets one.
  const unsigned threads = nblocks < 4 * sms ? 32 : 128;
  // Resident CTAs, asked for once: every device here is the same chip.
  static std::atomic<int> resident[2];
  int occ = resident[threads == 32].load(std::memory_order_relaxed);
  if (occ == 0) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, elementwise_planes_kernel<E, F>, threads, 0);
    if (e != cudaSuccess) return e;
    resident[threads == 32].store(occ, std::memory_order_relaxed);
  }
  const uint64_t want = (nblocks + threads / 32 - 1) / (threads / 32), cap = sms * static_cast<uint64_t>(occ < 1 ? 1 : occ);
  elementwise_planes_kernel<E, F>
      <<<static_cast<unsigned>(want < cap ? want : cap), threads, 0, s>>>(dst, a, b, len, head, nvec);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_elementwise_planes(int field, uint8_t* dst, const uint8_t* a, const uint8_t* b, uint64_t len,
                                      uint32_t head, uint64_t nvec, cudaStream_t s) {
  switch (field) {
    case kGf8B: return launch<1, kPoly1B>(dst, a, b, len, head, nvec, s);
    case kGf8D: return launch<1, kPoly1D>(dst, a, b, len, head, nvec, s);
    case kGf16: return launch<2, kPoly1B>(dst, a, b, len, head, nvec, s);
    case kGf32: return launch<4, kPoly1B>(dst, a, b, len, head, nvec, s);
    case kGf64: return launch<8, kPoly1B>(dst, a, b, len, head, nvec, s);
    case kFp8: return launch<1, kFanPaar>(dst, a, b, len, head, nvec, s);
    case kFp16: return launch<2, kFanPaar>(dst, a, b, len, head, nvec, s);
    case kFp32: return launch<4, kFanPaar>(dst, a, b, len, head, nvec, s);
    case kFp64: return launch<8, kFanPaar>(dst, a, b, len, head, nvec, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fgfc
