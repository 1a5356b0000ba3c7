// fast_core.cuh -- device building blocks shared by the single-call kernels
// (kernels.cu) and the persistent batch kernels (batch.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "internal.hpp"

namespace fgfc {

extern __shared__ __align__(16) uint8_t g_smem[];

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) {
  return __byte_perm(a, b, s);
}

__device__ __forceinline__ uint32_t lds_at(uint32_t off) {
  return *reinterpret_cast<const uint32_t*>(g_smem + off);
}

// Shifts by constants, MUL: on the multiply pipe. The bit-plane and tower-table
// kernels are bound by the ALU pipe (shifts, logic, permutes) with the FMA pipe
// nearly idle, and the compiler leaves right shifts and part of the left ones on
// the former. A multiplier it cannot see to be a power of two (grids are one
// CTA high, so gridDim.y is 1) makes x << s a product and x >> s the high half
// of one.
template <bool MUL>
struct Shift {
  uint32_t one;
  __device__ __forceinline__ Shift() : one(MUL ? gridDim.y : 1u) {}
  __device__ __forceinline__ uint32_t shl(uint32_t x, int s) const { return MUL ? x * (one << s) : x << s; }
  __device__ __forceinline__ uint32_t shr(uint32_t x, int s) const { return MUL ? __umulhi(x, one << (32 - s)) : x >> s; }
};

// Source loads: read-only path without L1 allocation (sources are read once).
__device__ __forceinline__ uint4 ldg16(const uint8_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// Pull a line into L2 ahead of its load (the next grid-stride iteration's
// column); this keeps more DRAM requests in flight than the registers of
// 1024-thread CTAs allow.
__device__ __forceinline__ void prefetch_l2(const uint8_t* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---------------------------------------------------------------- byte-table layout
//
// Gf8 fields with at most 4 rows (one table group) and a compile-time number
// of sources K. The first ones get a full 256-entry product table (one
// lookup per source byte, 32 KiB: 256 rows of 32 lane copies). The rest use
// single-copy 32-word tables after them, as lut.cuh does: five lookups for
// three sources, two for one (nibble tables with lane copies took two each).
// An address is a dot product of the data word (128 or 4 times one byte, plus
// the lane or nothing, beside the ALU pipe as in lut.cuh) plus an immediate.
constexpr int kFastMaxK = 14;
constexpr int kFastThreads = 1024;
// 2 to 10 sources: a thread holds two columns, the next one on its way while
// this one's lookups run (half the threads from 5 sources on, for the
// registers). More sources, and one alone, take 1024 threads and a prefetch of
// each thread's next column into L2. 16 MiB rows, 4 rows out, prefetch -> two
// columns, us: K = 6 33.2 -> 30.8, K = 8 38.8 -> 33.9, K = 10 47.7 -> 43.5; 4
// sources of 64 MiB into one row 55.9 -> 53.8, one into one 24.8 -> 29.1. Rows off
// the sources' boundaries (shift) hold more registers: 4 sources spill, and the
// batch kernels are slower from 4 on (4 rows, two columns -> prefetch: one call
// over 16 MiB of 4 sources 42.5 -> 40.2; 32 stripes of 1 MiB + 4 bytes, K = 4
// 112.8 -> 107.4, K = 6 148.4 -> 120.6, K = 8 164.2 -> 139.1, K = 10 179.2 ->
// 155.6; K = 2 with a plan per stripe 93.4 -> 98.2).
__host__ __device__ constexpr bool fast_pipe(int K, bool shift, bool batch) {
  return K >= 2 && K <= 10 && !(shift && (batch ? K >= 4 : K == 4));
}
__host__ __device__ constexpr int fast_threads(int K, bool shift, bool batch) {
  return K > 4 && fast_pipe(K, shift, batch) ? 512 : kFastThreads;
}

// Byte-table sources. Loads in flight live in what the tables leave of the 256
// KiB of L1: a seventh table (28 KiB left instead of 60) saves a lookup but cost
// one call over 16 MiB shards of RS(10,4) 52.1 us against 47.7, and fetching
// ahead with it cost batches 13 %. From 13 sources on four tables are better
// (K = 14: 73.8 -> 67.9 us), up to 12 six (K = 12: 57.2 against 59.4).
template <int K>
struct FastLayout {
  static constexpr int kMost = K <= 12 ? 6 : 4;
  static constexpr int NB = K < kMost ? K : kMost;        // byte-table sources
  static constexpr int NN = K - NB;                       // small-table sources
  static constexpr int N3 = NN / 3, N1 = NN % 3;          // threes, then single ones
  static constexpr uint32_t small = NB * 32768u;
  static constexpr uint32_t tables = small + N3 * 640u + N1 * 128u;
  static constexpr uint32_t smem = tables + K * kCompactWords * 4u;  // + compact staging
};

// Expand the compact tables of K sources (32 words each) into the byte-table
// layout. `tables` is a device pointer, or null to read `inl` (launch
// parameters). The compact words are staged in shared memory first (one
// independent load per thread) and every byte-table entry's 32 lane copies are
// written as 8 identical 16-byte stores.
template <int K>
__device__ __forceinline__ void fill_fast(const uint32_t* tables, const uint32_t* inl) {
  using L = FastLayout<K>;
  uint32_t* stage = reinterpret_cast<uint32_t*>(g_smem) + L::tables / 4;
  for (uint32_t i = threadIdx.x; i < K * kCompactWords; i += blockDim.x) {
    stage[i] = tables ? __ldg(tables + i) : inl[i];
  }
  __syncthreads();
  // byte tables: word index = t * 8192 + x * 32 + lane
  uint4* st4 = reinterpret_cast<uint4*>(g_smem);
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < L::NB * 2048u; i += blockDim.x) {
    const uint32_t t = i >> 11, x = (i >> 3) & 255u, q = i & 7u;
    const uint32_t v = stage[t * kCompactWords + (x & 15u)] ^ stage[t * kCompactWords + 16u + (x >> 4)];
    st4[t * 2048u + x * 8u + q] = make_uint4(v, v, v, v);
  }
  if constexpr (L::NN > 0) {
    // small tables: the words of one table are its 5- (or 4-) bit index
    uint32_t* out = reinterpret_cast<uint32_t*>(g_smem + L::small);
    for (uint32_t i = threadIdx.x; i < L::N3 * 160u + L::N1 * 32u; i += blockDim.x) {
      const uint32_t n = i & 31u;
      if (i < L::N3 * 160u) {
        const uint32_t q = i / 32u % 5u;
        const uint32_t* a = stage + (L::NB + 3u * (i / 160u)) * kCompactWords;  // source 0; 1 and 2 follow
        uint32_t v;
        if (q < 3)  // low 5 bits of source q
          v = a[q * kCompactWords + (n & 15u)] ^ a[q * kCompactWords + 16u + (n >> 4)];
        else if (q == 3)  // bits 5..7 of source 0, 5 and 6 of source 1
          v = a[16u + 2u * (n & 7u)] ^ a[kCompactWords + 16u + 2u * (n >> 3)];
        else  // bits 5..7 of source 2, 7 of source 1
          v = a[2u * kCompactWords + 16u + 2u * (n & 7u)] ^ a[kCompactWords + 16u + (n & 8u)];
        out[i] = v;
      } else {
        out[i] = stage[(L::NB + 3u * L::N3 + (i - L::N3 * 160u) / 32u) * kCompactWords + n];
      }
    }
  }
  __syncthreads();
}

// base + M times byte b of x, beside the ALU pipe (lut.cuh: lut_addr).
template <uint32_t M>
__device__ __forceinline__ uint32_t byte_addr(uint32_t x, uint32_t base, int b) {
  return __dp4a(x, M << (8 * b), base);
}

// Fold NW words (4 bytes each, byte b of word q is element 4q + b) of each
// of the K sources into acc (acc[e] = products for rows 0..3 of element e).
// lane4: 4 times the lane.
template <int K, int NW>
__device__ __forceinline__ void fast_fold(const uint32_t (&w)[K][NW], uint32_t (&acc)[4 * NW], uint32_t lane4) {
  using L = FastLayout<K>;
#pragma unroll
  for (int t = 0; t < L::NB; t += 2) {
#pragma unroll
    for (int q = 0; q < NW; ++q)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        uint32_t v = lds_at(byte_addr<128>(w[t][q], lane4, b) + t * 32768u);
        if (t + 1 < L::NB) v ^= lds_at(byte_addr<128>(w[t + 1][q], lane4, b) + (t + 1) * 32768u);
        acc[4 * q + b] ^= v;
      }
  }
#pragma unroll
  for (int i = 0; i < L::N3; ++i) {
    const int t = L::NB + 3 * i;
#pragma unroll
    for (int q = 0; q < NW; ++q) {
      const uint32_t i0 = w[t][q] & 0x1F1F1F1Fu, i1 = w[t + 1][q] & 0x1F1F1F1Fu, i2 = w[t + 2][q] & 0x1F1F1F1Fu;
      const uint32_t i3 = ((w[t][q] >> 3) & 0x1C1C1C1Cu) | (w[t + 1][q] & 0x60606060u);
      const uint32_t i4 = ((w[t + 2][q] >> 3) & 0x1C1C1C1Cu) | ((w[t + 1][q] >> 2) & 0x20202020u);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        constexpr uint32_t o = L::small;
        acc[4 * q + b] ^= lds_at(byte_addr<4>(i0, 0, b) + o + i * 640u) ^ lds_at(byte_addr<4>(i1, 0, b) + o + i * 640u + 128u);
        acc[4 * q + b] ^= lds_at(byte_addr<4>(i2, 0, b) + o + i * 640u + 256u) ^
                          lds_at(byte_addr<1>(i3, 0, b) + o + i * 640u + 384u);
        acc[4 * q + b] ^= lds_at(byte_addr<1>(i4, 0, b) + o + i * 640u + 512u);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < L::N1; ++i) {
    const int t = L::NB + 3 * L::N3 + i;
#pragma unroll
    for (int q = 0; q < NW; ++q) {
      const uint32_t i0 = w[t][q] & 0x0F0F0F0Fu, i1 = (w[t][q] >> 4) & 0x0F0F0F0Fu;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        constexpr uint32_t o = L::small + L::N3 * 640u;
        acc[4 * q + b] ^= lds_at(byte_addr<4>(i0, 0, b) + o + i * 128u) ^ lds_at(byte_addr<4>(i1, 0, b) + o + i * 128u + 64u);
      }
    }
  }
}

// 16 bytes of each of the K sources at byte off.
template <int K>
__device__ __forceinline__ void fast_load(const uint8_t* const* src, uint64_t off, uint32_t (&w)[K][4]) {
#pragma unroll
  for (int t = 0; t < K; ++t) {
    const uint4 x = ldg16(src[t] + off);
    w[t][0] = x.x;
    w[t][1] = x.y;
    w[t][2] = x.z;
    w[t][3] = x.w;
  }
}

// Row rr (0..3) of one output word from 4 element accumulators (4x4 byte
// transpose: acc[e] holds rows 0..3 of element e).
__device__ __forceinline__ uint32_t row_word4(const uint32_t* acc, int rr) {
  const uint32_t s01 = prmt(acc[0], acc[1], rr < 2 ? 0x5140u : 0x7362u);
  const uint32_t s23 = prmt(acc[2], acc[3], rr < 2 ? 0x5140u : 0x7362u);
  return prmt(s01, s23, (rr & 1) ? 0x7632u : 0x5410u);
}

// Group gi of the 4-byte groups before (head) and after the 16-byte columns of a
// job: nb bytes at *off.
__device__ __forceinline__ int fast_group(uint64_t len, uint64_t head, uint64_t nvec, uint64_t gi, uint64_t* off) {
  const uint64_t tail0 = head + nvec * 16u, n0 = (head + 3) / 4;
  *off = gi < n0 ? 4 * gi : tail0 + 4 * (gi - n0);
  const uint64_t end = gi < n0 ? head : len;
  return static_cast<int>(end - *off < 4 ? end - *off : 4);
}
__host__ __device__ inline uint64_t fast_groups(uint64_t len, uint64_t head, uint64_t nvec) {
  return (head + 3) / 4 + (len - head - 16 * nvec + 3) / 4;
}

// Bytes [off, off + nb) of the rows, one thread, bytewise.
template <int K>
__device__ __forceinline__ void fast_bytes(const uint8_t* const* src, uint8_t* const* dst, uint32_t nrows, uint64_t off,
                                           int nb, bool ovr, uint32_t lane4) {
  uint32_t w[K][1];
#pragma unroll
  for (int t = 0; t < K; ++t) {
    uint32_t x = 0;
    for (int b = 0; b < nb; ++b) x |= static_cast<uint32_t>(src[t][off + b]) << (8 * b);
    w[t][0] = x;
  }
  uint32_t acc[4] = {0, 0, 0, 0};
  fast_fold<K, 1>(w, acc, lane4);
  for (uint32_t rr = 0; rr < nrows; ++rr) {
    const uint32_t o = row_word4(acc, static_cast<int>(rr));
    uint8_t* d = dst[rr] + off;
    for (int b = 0; b < nb; ++b) {
      const uint8_t v = static_cast<uint8_t>(o >> (8 * b));
      d[b] = ovr ? v : static_cast<uint8_t>(d[b] ^ v);
    }
  }
}

// ---------------------------------------------------------------- row stores
//
// The vector paths compute 16-byte columns in the alignment of the sources.
// A destination row may start anywhere (contiguous rows of any length put
// row j at j * row_len). When a column's destination is dl = addr & 15 bytes
// past a 16-byte boundary, each lane writes the aligned 16 bytes that end
// inside its column, spliced from the previous lane's column (one warp
// shuffle per word) and its own; the ends of a run of contiguous columns are
// written bytewise. Every byte is written by exactly one lane. All 32 lanes
// of the warp must call store_vec16 together; lanes without a column pass
// valid = false.

constexpr unsigned kFullWarp = 0xffffffffu;

// Bytes [s, s + 16) of the 32-byte concatenation P || V, 0 < s < 16.
__device__ __forceinline__ uint4 splice16(const uint4& P, const uint4& V, uint32_t s) {
  uint32_t c0, c1, c2, c3, c4;
  switch (s >> 2) {
    case 0: c0 = P.x; c1 = P.y; c2 = P.z; c3 = P.w; c4 = V.x; break;
    case 1: c0 = P.y; c1 = P.z; c2 = P.w; c3 = V.x; c4 = V.y; break;
    case 2: c0 = P.z; c1 = P.w; c2 = V.x; c3 = V.y; c4 = V.z; break;
    default: c0 = P.w; c1 = V.x; c2 = V.y; c3 = V.z; c4 = V.w; break;
  }
  const uint32_t r = (s & 3u) * 8u;
  return make_uint4(__funnelshift_r(c0, c1, r), __funnelshift_r(c1, c2, r), __funnelshift_r(c2, c3, r),
                    __funnelshift_r(c3, c4, r));
}

// Bytes [b0, b1) of V to p[0 .. b1 - b0), one byte store each.
__device__ __forceinline__ void put_bytes(uint8_t* p, const uint4& V, uint32_t b0, uint32_t b1, bool ovr) {
  const uint32_t w[4] = {V.x, V.y, V.z, V.w};
#pragma unroll
  for (uint32_t b = 0; b < 16; ++b) {
    if (b < b0 || b >= b1) continue;
    const uint8_t v = static_cast<uint8_t>(w[b >> 2] >> (8 * (b & 3u)));
    uint8_t* q = p + (b - b0);
    *q = ovr ? v : static_cast<uint8_t>(*q ^ v);
  }
}

__device__ __forceinline__ void put16(uint8_t* p, uint4 o, bool ovr) {
  uint4* dp = reinterpret_cast<uint4*>(p);
  if (!ovr) {
    const uint4 d = *dp;
    o.x ^= d.x;
    o.y ^= d.y;
    o.z ^= d.z;
    o.w ^= d.w;
  }
  *dp = o;
}

// Store the 16-byte column o at p (any alignment); accumulate unless ovr.
__device__ __forceinline__ void store_vec16(uint8_t* p, const uint4& o, bool valid, bool ovr) {
  const uint64_t a = reinterpret_cast<uint64_t>(p);
  const uint32_t dl = static_cast<uint32_t>(a) & 15u;
  if (__all_sync(kFullWarp, !valid || dl == 0)) {
    if (valid) put16(p, o, ovr);
    return;
  }
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t ap = __shfl_up_sync(kFullWarp, a, 1);
  const uint64_t an = __shfl_down_sync(kFullWarp, a, 1);
  const int vp = __shfl_up_sync(kFullWarp, valid ? 1 : 0, 1);
  const int vn = __shfl_down_sync(kFullWarp, valid ? 1 : 0, 1);
  uint4 P;
  P.x = __shfl_up_sync(kFullWarp, o.x, 1);
  P.y = __shfl_up_sync(kFullWarp, o.y, 1);
  P.z = __shfl_up_sync(kFullWarp, o.z, 1);
  P.w = __shfl_up_sync(kFullWarp, o.w, 1);
  if (!valid) return;
  if (dl == 0) {
    put16(p, o, ovr);
    return;
  }
  const bool prev_ok = lane > 0 && vp && ap + 16 == a;
  const bool next_ok = lane < 31 && vn && an == a + 16;
  const uint32_t s = 16u - dl;
  if (prev_ok)
    put16(p - dl, splice16(P, o, s), ovr);  // [p - dl, p + s): previous column's tail, then ours
  else
    put_bytes(p, o, 0, s, ovr);
  if (!next_ok) put_bytes(p + s, o, s, 16, ovr);
}

// Store one 16-byte column of up to 4 rows whose destinations share the
// sources' alignment; accumulate unless overwriting.
__device__ __forceinline__ void store_col4(const uint32_t (&acc)[16], uint8_t* const* dst, uint32_t nrows,
                                           uint64_t off, bool ovr) {
#pragma unroll
  for (int rr = 0; rr < 4; ++rr) {
    if (rr >= static_cast<int>(nrows)) break;
    uint4 o;
    o.x = row_word4(&acc[0], rr);
    o.y = row_word4(&acc[4], rr);
    o.z = row_word4(&acc[8], rr);
    o.w = row_word4(&acc[12], rr);
    put16(dst[rr] + off, o, ovr);
  }
}

// The same for rows at any offset. Called by every lane of the warp;
// `valid` marks lanes holding a column.
__device__ __forceinline__ void store_col4_any(const uint32_t (&acc)[16], uint8_t* const* dst, uint32_t nrows,
                                               uint64_t off, bool ovr, bool valid) {
#pragma unroll
  for (int rr = 0; rr < 4; ++rr) {
    uint4 o;
    o.x = row_word4(&acc[0], rr);
    o.y = row_word4(&acc[4], rr);
    o.z = row_word4(&acc[8], rr);
    o.w = row_word4(&acc[12], rr);
    const bool rv = valid && rr < static_cast<int>(nrows);
    store_vec16(rv ? dst[rr] + off : nullptr, o, rv, ovr);
  }
}

}  // namespace fgfc
