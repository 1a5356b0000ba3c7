// lut.cuh -- the table kernels for every field and shape of the matrix ops:
// rows[j] (^)= XOR_t c[t][j] * src_t.
//
// Lookups. A product by a constant is linear over GF(2), so a 4-byte output
// word is the XOR of table words indexed by a few input bits. A 32-word table
// is exactly one row of the 32 shared-memory banks: lanes that look up
// different words hit different banks and lanes that look up the same word are
// served by one broadcast, so a warp's 32 lookups never conflict whatever the
// data, with a single 128-byte copy of the table. Five index bits per lookup
// is therefore the widest conflict-free table: one bit more doubles the
// wavefronts, and copies per lane (32 x 128 bytes per nibble pair) hold a kernel
// to one CTA per SM and a 1.5 us fill. Three sources
// are folded together: 24 bits of one byte position of three sources take five
// lookups (each byte's low 5 bits, then the 3 + 2 and 1 + 3 bits left over)
// where nibble tables take six.
//
// Towers. Each level of a tower halves the element, c = c0 + c1 X and
// x = x0 + x1 X, and needs three half-products (Karatsuba) A = c0 x0,
// B = c1 x1, C = (c0 + c1)(x0 + x1), with a linear fix-up of the sums over
// all sources at the end:
//   Gf16/32/64 (X^2 = X + beta):      lo = A + beta B, hi = A + C
//   Fan-Paar   (X^2 = alpha X + 1):   lo = A + B,      hi = A + C + B + alpha B.
// With LEV levels the leaves are H = E >> LEV bytes wide and a table word holds
// the leaf products of 4 / H rows. More levels mean fewer lookups per row but
// need enough rows to fill the word and enough sources to carry the fix-up, which
// is the rule of lut_shape(). Short rows of 8-byte elements run wide.cu.
//
// What bounds it: the lookups (one shared-memory wavefront each) and, with one
// word per product, the issue slots of the operations around them (address dot
// product, XOR, index masks). Measured on B200 against 16-word tables with 32 copies
// per lane (or unreplicated for 8-byte elements):
//   GF(2^64) RS(10,4), 16 MiB shards     308 -> 173 us (lookups per element 992 -> 459)
//   256 stripes of Gf8D and Gf16, k 4..32, m 1..8, 4 KiB .. 4 MiB, one batch
//                                        3240 -> 1320 us (more CTAs resident, no 216 KiB refills)
//   Gf8D RS(12,4), consecutive shards of 1000003 bytes: 24.1 -> 7.7 us (by single
//   bytes, by spliced 16-byte granules)
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "fast_core.cuh"
#include "internal.hpp"

namespace fgfc {

// ---------------------------------------------------------------- shapes

__host__ __device__ constexpr int pow3(int n) { return n <= 0 ? 1 : 3 * pow3(n - 1); }

template <int E, int LEV>
struct Lut {
  static constexpr int H = E >> LEV;          // leaf bytes
  static constexpr int NP = pow3(LEV);        // leaf products per element
  static constexpr int NV = NP * H;           // leaf input bytes per element
  static constexpr int NE = 16 / E;           // elements per 16-byte column
  static constexpr int NW = (NE * NV + 3) / 4;  // packed words of leaf input bytes per column
  static constexpr int NF = 16 / H;           // accumulator words per column after the fix-up
  // Index shifts on the multiply pipe: GF(2^64) RS(10,4), 16 MiB, 204 -> 173 us;
  // level or worse for the other widths.
  static constexpr bool kMulShift = E == 8;
  static constexpr bool kDirect = LEV == 0 && E > 1;  // no split

  // element and leaf byte (product * H + byte) of byte b of packed word w;
  // elem() < 0: no byte there
  static __host__ __device__ constexpr int elem(int w, int b) {
    if (E == 1) return 4 * w + b;
    if (E == 2) return LEV == 0 ? 2 * w + b / 2 : 4 * (w & 1) + b;
    if (E == 4) return LEV == 0 ? w : LEV == 1 ? 2 * (w & 1) + b / 2 : b;
    if (LEV <= 1) return w & 1;
    if (LEV == 2) return b / 2;
    if (w < 9) return b / 2;
    return w == 13 && b >= 2 ? -1 : b & 1;
  }
  static __host__ __device__ constexpr int vb(int w, int b) {
    if (E == 1) return 0;
    if (E == 2) return LEV == 0 ? b & 1 : w >> 1;
    if (E == 4) return LEV == 0 ? b : LEV == 1 ? 2 * (w >> 1) + (b & 1) : w;
    if (LEV <= 1) return 4 * (w >> 1) + b;
    if (LEV == 2) return 2 * w + (b & 1);
    if (w < 9) return 3 * w + (b & 1);
    return 3 * (2 * (w - 9) + b / 2) + 2;
  }

  // The packed words of one 16-byte column.
  static __device__ __forceinline__ void expand(const uint4& x, uint32_t (&v)[NW]) {
    if constexpr (E == 1 || (E <= 4 && LEV == 0)) {
      v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    } else if constexpr (E == 2) {  // [lo bytes x 4], [lo], [hi], [hi], [lo + hi], [lo + hi]
      v[0] = prmt(x.x, x.y, 0x6420u), v[1] = prmt(x.z, x.w, 0x6420u);
      v[2] = prmt(x.x, x.y, 0x7531u), v[3] = prmt(x.z, x.w, 0x7531u);
      v[4] = v[0] ^ v[2], v[5] = v[1] ^ v[3];
    } else if constexpr (E == 4 && LEV == 1) {  // 16-bit halves of two elements per word
      v[0] = prmt(x.x, x.y, 0x5410u), v[1] = prmt(x.z, x.w, 0x5410u);
      v[2] = prmt(x.x, x.y, 0x7632u), v[3] = prmt(x.z, x.w, 0x7632u);
      v[4] = v[0] ^ v[2], v[5] = v[1] ^ v[3];
    } else if constexpr (E == 4) {  // byte planes of the 4 elements, products in tree order
      const uint32_t a = prmt(x.x, x.y, 0x5140u), b = prmt(x.z, x.w, 0x5140u);
      const uint32_t c = prmt(x.x, x.y, 0x7362u), d = prmt(x.z, x.w, 0x7362u);
      v[0] = prmt(a, b, 0x5410u), v[1] = prmt(a, b, 0x7632u);
      v[3] = prmt(c, d, 0x5410u), v[4] = prmt(c, d, 0x7632u);
      v[2] = v[0] ^ v[1], v[5] = v[3] ^ v[4];
      v[6] = v[0] ^ v[3], v[7] = v[1] ^ v[4], v[8] = v[2] ^ v[5];
    } else if constexpr (LEV <= 1) {  // 8-byte elements: lo, lo, hi, hi, lo + hi, lo + hi
      v[0] = x.x, v[1] = x.z, v[2] = x.y, v[3] = x.w;
      if constexpr (LEV == 1) v[4] = x.x ^ x.y, v[5] = x.z ^ x.w;
    } else {  // 16-bit quarters of the two elements, 9 products in tree order
      v[0] = prmt(x.x, x.z, 0x5410u), v[1] = prmt(x.x, x.z, 0x7632u);
      v[3] = prmt(x.y, x.w, 0x5410u), v[4] = prmt(x.y, x.w, 0x7632u);
      v[2] = v[0] ^ v[1], v[5] = v[3] ^ v[4];
      v[6] = v[0] ^ v[3], v[7] = v[1] ^ v[4], v[8] = v[2] ^ v[5];
      if constexpr (LEV == 3) {  // byte sums of the 9 halves, two halves per word
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const uint32_t p = v[2 * i] ^ (v[2 * i] >> 8);
          const uint32_t q = i < 4 ? v[2 * i + 1] ^ (v[2 * i + 1] >> 8) : 0u;
          v[9 + i] = prmt(p, q, 0x6420u);
        }
      }
    }
  }
};

// Shared-memory tables: per 3 sources five 32-word tables for each (leaf
// byte, output word), then two 16-word nibble tables per (leaf byte, output
// word) for each of the k % 3 sources left. An address is the block's base plus
// 4 times the index (lut_addr) plus an immediate.
template <int NV, int W>
struct LutSmem {
  static constexpr uint32_t block3 = (NV * W * 640u + 255u) / 256u * 256u;
  static constexpr uint32_t block1 = (NV * W * 128u + 255u) / 256u * 256u;
};

// Direct shapes of several words per element (2- and 4-byte fields) serve calls of
// one or two sources: no groups of three.
template <class L, int W>
constexpr bool kLutFewSources = L::kDirect && W > 1;

// ---------------------------------------------------------------- table fill

// Tables of k sources from their images (8 words per (source, leaf byte,
// output word): the word for each single input bit).
template <class L, int W>
__device__ __forceinline__ void lut_fill(const uint32_t* img, uint32_t k) {
  using S = LutSmem<L::NV, W>;
  constexpr uint32_t NS = L::NV * W;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint32_t m[5];
#pragma unroll
  for (int b = 0; b < 5; ++b) m[b] = 0u - ((lane >> b) & 1u);
  const uint4* im = reinterpret_cast<const uint4*>(img);
  const uint32_t nt = kLutFewSources<L, W> ? 0 : k / 3u, tasks = nt * NS;
#pragma unroll 2
  for (uint32_t i = warp; i < tasks; i += nwarps) {
    const uint32_t tr = i / NS, s = i - tr * NS;
    const uint4* p = im + 2u * (3u * tr * NS + s);
    const uint4 a = p[0], a2 = p[1], b = p[2 * NS], b2 = p[2 * NS + 1], c = p[4 * NS], c2 = p[4 * NS + 1];
    uint32_t* out = reinterpret_cast<uint32_t*>(g_smem + tr * S::block3 + s * 640u) + lane;
    out[0] = (a.x & m[0]) ^ (a.y & m[1]) ^ (a.z & m[2]) ^ (a.w & m[3]) ^ (a2.x & m[4]);
    out[32] = (b.x & m[0]) ^ (b.y & m[1]) ^ (b.z & m[2]) ^ (b.w & m[3]) ^ (b2.x & m[4]);
    out[64] = (c.x & m[0]) ^ (c.y & m[1]) ^ (c.z & m[2]) ^ (c.w & m[3]) ^ (c2.x & m[4]);
    out[96] = (a2.y & m[0]) ^ (a2.z & m[1]) ^ (a2.w & m[2]) ^ (b2.y & m[3]) ^ (b2.z & m[4]);
    out[128] = (c2.y & m[0]) ^ (c2.z & m[1]) ^ (c2.w & m[2]) ^ (b2.w & m[3]);
  }
  const uint32_t rest = k - 3u * nt;
  for (uint32_t i = warp; i < rest * NS; i += nwarps) {
    const uint32_t r = i / NS, s = i - r * NS;
    const uint4* p = im + 2u * ((3u * nt + r) * NS + s);
    const uint4 v = p[lane >> 4];  // lanes 0..15: low nibble, 16..31: high nibble
    uint32_t* out = reinterpret_cast<uint32_t*>(g_smem + nt * S::block3 + r * S::block1 + s * 128u) + lane;
    *out = (v.x & m[0]) ^ (v.y & m[1]) ^ (v.z & m[2]) ^ (v.w & m[3]);
  }
}

// ---------------------------------------------------------------- folds

// Accumulators: the word of leaf product P, output word g, element e.
template <class L, int W>
struct LutAcc {
  uint32_t a[L::NP][W][L::NE];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int p = 0; p < L::NP; ++p)
#pragma unroll
      for (int g = 0; g < W; ++g)
#pragma unroll
        for (int e = 0; e < L::NE; ++e) a[p][g][e] = 0;
  }
};

// base + M times byte b of x. A dot product of bytes with one nonzero factor:
// it runs beside the ALU pipe, which a PRMT per lookup kept at 80 % (PRMT ->
// dot product: GF(2^64) RS(10,4) 16 MiB 190 -> 173 us, Gf32 RS(16,4) 8 MiB
// 86 -> 79, Gf16 RS(12,4) 4 MiB 27.8 -> 24.8, Gf8D RS(20,4) 4 MiB 29.2 -> 28.5).
template <uint32_t M>
__device__ __forceinline__ uint32_t lut_addr(uint32_t x, uint32_t base, int b) {
  return __dp4a(x, M << (8 * b), base);
}

// Three sources whose tables start at `base`.
template <class L, int W>
__device__ __forceinline__ void lut_fold3(const uint4& c0, const uint4& c1, const uint4& c2, uint32_t base,
                                          LutAcc<L, W>& A) {
  uint32_t v0[L::NW], v1[L::NW], v2[L::NW];
  L::expand(c0, v0);
  L::expand(c1, v1);
  L::expand(c2, v2);
  const Shift<L::kMulShift> sh;
#pragma unroll
  for (int w = 0; w < L::NW; ++w) {
    const uint32_t i0 = v0[w] & 0x1F1F1F1Fu, i1 = v1[w] & 0x1F1F1F1Fu, i2 = v2[w] & 0x1F1F1F1Fu;
    const uint32_t i3 = (sh.shr(v0[w], 3) & 0x1C1C1C1Cu) | (v1[w] & 0x60606060u);
    const uint32_t i4 = (sh.shr(v2[w], 3) & 0x1C1C1C1Cu) | (sh.shr(v1[w], 2) & 0x20202020u);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (L::elem(w, b) < 0) continue;
      const int e = L::elem(w, b), vb = L::vb(w, b), p = vb / L::H;
      const uint32_t q0 = lut_addr<4>(i0, base, b), q1 = lut_addr<4>(i1, base, b), q2 = lut_addr<4>(i2, base, b),
                     q3 = lut_addr<1>(i3, base, b), q4 = lut_addr<1>(i4, base, b);
#pragma unroll
      for (int g = 0; g < W; ++g) {
        const uint32_t o = (vb * W + g) * 640u;
        A.a[p][g][e] ^= lds_at(q0 + o) ^ lds_at(q1 + o + 128u);
        A.a[p][g][e] ^= lds_at(q2 + o + 256u) ^ lds_at(q3 + o + 384u);
        A.a[p][g][e] ^= lds_at(q4 + o + 512u);
      }
    }
  }
}

// One source with nibble tables at `base`.
template <class L, int W>
__device__ __forceinline__ void lut_fold1(const uint4& c0, uint32_t base, LutAcc<L, W>& A) {
  uint32_t v0[L::NW];
  L::expand(c0, v0);
  const Shift<L::kMulShift> sh;
#pragma unroll
  for (int w = 0; w < L::NW; ++w) {
    const uint32_t i0 = v0[w] & 0x0F0F0F0Fu, i1 = sh.shr(v0[w], 2) & 0x3C3C3C3Cu;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (L::elem(w, b) < 0) continue;
      const int e = L::elem(w, b), vb = L::vb(w, b), p = vb / L::H;
      const uint32_t q0 = lut_addr<4>(i0, base, b), q1 = lut_addr<1>(i1, base, b);
#pragma unroll
      for (int g = 0; g < W; ++g) {
        const uint32_t o = (vb * W + g) * 128u;
        A.a[p][g][e] ^= lds_at(q0 + o) ^ lds_at(q1 + o + 64u);
      }
    }
  }
}

// ---------------------------------------------------------------- tower fix-ups

// beta and alpha of the levels, on words holding 4 / H lanes of H bytes.

// x^5 = 0x20 times every byte over x^8 + x^4 + x^3 + x + 1: with t = v >> 3
// the part that overflows is t (x^4 + x^3 + x + 1), whose own overflow (the
// top bit of t, 0x80 of v) folds in as the polynomial again.
__device__ __forceinline__ uint32_t lut_mul20(uint32_t v) {
  const uint32_t t = (v >> 3) & 0x1F1F1F1Fu;
  const uint32_t r = ((v << 5) & 0xE0E0E0E0u) ^ t ^ (t << 1) ^ (t << 3) ^ ((t & 0x0F0F0F0Fu) << 4);
  return r ^ (((v >> 7) & 0x01010101u) * 0x1Bu);
}

// The Fan-Paar byte level's generator times every byte: one step of
// alpha (a0 + a1 X) = a1 + (a0 + alpha' a1) X per level.
__device__ __forceinline__ uint32_t lut_fp_alpha8(uint32_t v) {
  const uint32_t h = (v >> 4) & 0x0F0F0F0Fu;                  // a1 of the byte
  const uint32_t q = (h >> 2) & 0x03030303u;                  // a1 of the nibble
  const uint32_t c = (q >> 1) & 0x01010101u;
  const uint32_t p = c | (((q ^ c) & 0x01010101u) << 1);      // alpha2 q = (q1, q0 + q1)
  const uint32_t n = q | (((h & 0x03030303u) ^ p) << 2);      // alpha4 h
  return h | (((v & 0x0F0F0F0Fu) ^ n) << 4);
}

// One lane-packed word: lanes of H bytes.
template <int H, bool FP>
__device__ __forceinline__ uint32_t lut_const1(uint32_t v) {
  if constexpr (H == 1) {
    return FP ? lut_fp_alpha8(v) : lut_mul20(v);
  } else if constexpr (H == 2) {
    const uint32_t hi = (v >> 8) & 0x00FF00FFu;
    if (FP)  // (b0, b1) -> (b1, b0 + alpha b1)
      return hi | (((v << 8) ^ (lut_fp_alpha8(hi) << 8)) & 0xFF00FF00u);
    // (b0, b1) -> beta (beta b1, b0 + b1)
    const uint32_t w = lut_mul20(hi | (((v << 8) ^ v) & 0xFF00FF00u));
    return (w & 0xFF00FF00u) | (lut_mul20(w) & 0x00FF00FFu);
  } else {
    const uint32_t hi = v >> 16;
    if (FP) return hi | (((v << 16) ^ (lut_const1<2, true>(hi) << 16)) & 0xFFFF0000u);
    const uint32_t w = lut_const1<2, false>(hi | ((v << 16) ^ (v & 0xFFFF0000u)));
    return (w & 0xFFFF0000u) | (lut_const1<2, false>(w) & 0x0000FFFFu);
  }
}

// The level's constant (beta, or alpha for Fan-Paar) times a value of N words.
template <int H, int N, bool FP>
__device__ __forceinline__ void lut_const(const uint32_t* v, uint32_t* out) {
  if constexpr (N == 1) {
    out[0] = lut_const1<H, FP>(v[0]);
  } else {
    constexpr int M = N / 2;
    if constexpr (FP) {
      uint32_t t[M];
      lut_const<H, M, FP>(v + M, t);
#pragma unroll
      for (int i = 0; i < M; ++i) {
        out[i] = v[M + i];
        out[M + i] = v[i] ^ t[i];
      }
    } else {
      uint32_t s[M], t[M];
      lut_const<H, M, FP>(v + M, t);
      lut_const<H, M, FP>(t, out);
#pragma unroll
      for (int i = 0; i < M; ++i) s[i] = v[i] ^ v[M + i];
      lut_const<H, M, FP>(s, out + M);
    }
  }
}

// Leaf products in tree order (3^LEV words) to the element (2^LEV words).
template <int H, int LEV, bool FP>
__device__ __forceinline__ void lut_combine(const uint32_t* leaf, uint32_t* out) {
  if constexpr (LEV == 0) {
    out[0] = leaf[0];
  } else {
    constexpr int N = 1 << (LEV - 1), P = pow3(LEV - 1);
    uint32_t a[N], b[N], c[N], t[N];
    lut_combine<H, LEV - 1, FP>(leaf, a);
    lut_combine<H, LEV - 1, FP>(leaf + P, b);
    lut_combine<H, LEV - 1, FP>(leaf + 2 * P, c);
    lut_const<H, N, FP>(b, t);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      out[i] = a[i] ^ (FP ? b[i] : t[i]);
      out[N + i] = a[i] ^ c[i] ^ (FP ? b[i] ^ t[i] : 0u);
    }
  }
}

// A column's accumulators as words in byte order: f[g][e * E / H + i].
template <class L, int W, int LEV>
__device__ __forceinline__ void lut_finish(const LutAcc<L, W>& A, uint32_t (&f)[W][L::NF], bool fp) {
  if constexpr (LEV == 0) {
#pragma unroll
    for (int g = 0; g < W; ++g)
#pragma unroll
      for (int e = 0; e < L::NE; ++e) f[g][e] = A.a[0][g][e];
  } else {
    constexpr int N = 1 << LEV;
#pragma unroll
    for (int g = 0; g < W; ++g)
#pragma unroll
      for (int e = 0; e < L::NE; ++e) {
        uint32_t leaf[L::NP];
#pragma unroll
        for (int p = 0; p < L::NP; ++p) leaf[p] = A.a[p][g][e];
        if (fp)
          lut_combine<L::H, LEV, true>(leaf, &f[g][e * N]);
        else
          lut_combine<L::H, LEV, false>(leaf, &f[g][e * N]);
      }
  }
}

// Row r (of the 4 / H in output word g) of a finished column.
template <class L>
__device__ __forceinline__ uint4 lut_row(const uint32_t (&f)[L::NF], int r) {
  uint32_t o[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if constexpr (L::H == 1)
      o[q] = row_word4(&f[4 * q], r);
    else if constexpr (L::H == 2)
      o[q] = prmt(f[2 * q], f[2 * q + 1], r ? 0x7632u : 0x5410u);
    else
      o[q] = f[q];
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// ---------------------------------------------------------------- one job

struct LutShared {
  const uint8_t* src[kMaxSrc];
  uint8_t* dst[kLutRows];
};

// Three sources' 16-byte columns on their way from memory.
struct LutAhead {
  uint4 c[3];
};

// Does a shape fetch the next column's first sources during the last lookups of
// this one (not with unaligned sources)? It hides the fetch where 16 to 24 warps
// an SM do not (us, without -> with: Gf16 RS(32,8) 16 MiB 355 -> 339, Gf32
// RS(16,4) 8 MiB 91 -> 86, Gf8D RS(32,12) 4 MiB 103 -> 99); shapes of few
// accumulators keep their warps instead, and two rows of 8-byte elements (18)
// lose (RS(8,2) 4 MiB 29.7 against 30.1).
template <class L, int W>
constexpr bool kLutAhead = L::NP * W * L::NE >= (L::NE == 2 ? 32 : 16);

// Fold all sources of one column. load(t) fetches source t's 16 bytes, fix(t, x)
// puts a fetch in place once it is needed. The fetches of the next three
// sources are in flight during the lookups.
template <class L, int W, class Load, class Fix>
__device__ __forceinline__ void lut_column(LutAcc<L, W>& A, uint32_t k, Load load, Fix fix) {
  using S = LutSmem<L::NV, W>;
  A.zero();
  const uint32_t nt = kLutFewSources<L, W> ? 0 : k / 3u;
  uint4 c0 = load(0u), c1, c2;
  c1 = c2 = make_uint4(0, 0, 0, 0);
  if (k > 1) c1 = load(1u);
  if (k > 2) c2 = load(2u);
  uint32_t base = 0;
  for (uint32_t i = 0; i < nt; ++i) {
    uint4 n0 = c0, n1 = c1, n2 = c2;
    const uint32_t t = 3u * i + 3u;
    if (t < k) n0 = load(t);
    if (t + 1u < k) n1 = load(t + 1u);
    if (t + 2u < k) n2 = load(t + 2u);
    lut_fold3<L, W>(fix(t - 3u, c0), fix(t - 2u, c1), fix(t - 1u, c2), base, A);
    c0 = n0, c1 = n1, c2 = n2;
    base += S::block3;
  }
  const uint32_t rest = k - 3u * nt;
  for (uint32_t r = 0; r < rest; ++r) {
    lut_fold1<L, W>(fix(3u * nt + r, c0), base, A);
    c0 = c1;
    base += S::block1;
  }
}

// The same for shapes that look ahead: on entry h holds this column's first
// three sources, on return the next column's, which next(t) fetches.
template <class L, int W, class Load, class Next, class Fix>
__device__ __forceinline__ void lut_column_ahead(LutAcc<L, W>& A, uint32_t k, LutAhead& h, Load load, Next next,
                                                 Fix fix) {
  using S = LutSmem<L::NV, W>;
  A.zero();
  const uint32_t nt = kLutFewSources<L, W> ? 0 : k / 3u, rest = k - 3u * nt;
  uint32_t base = 0;
  for (uint32_t i = 0; i < nt; ++i) {
    const uint32_t t = 3u * i;
    const uint4 x0 = fix(t, h.c[0]), x1 = fix(t + 1u, h.c[1]), x2 = fix(t + 2u, h.c[2]);
    if (t + 3u < k) {
#pragma unroll
      for (uint32_t j = 0; j < 3; ++j)
        if (t + 3u + j < k) h.c[j] = load(t + 3u + j);
    } else {
#pragma unroll
      for (uint32_t j = 0; j < 3; ++j) h.c[j] = next(j);
    }
    lut_fold3<L, W>(x0, x1, x2, base, A);
    base += S::block3;
  }
  if (rest) {
    const uint32_t t = 3u * nt;
    const uint4 x0 = fix(t, h.c[0]);
    uint4 x1 = x0;
    if (rest > 1) x1 = fix(t + 1u, h.c[1]);
#pragma unroll
    for (uint32_t j = 0; j < 3; ++j)
      if (j < k) h.c[j] = next(j);
    lut_fold1<L, W>(x0, base, A);
    if (rest > 1) lut_fold1<L, W>(x1, base + S::block1, A);
  }
}

struct LutAsIs {
  __device__ __forceinline__ uint4 operator()(uint32_t, const uint4& x) const { return x; }
};

// Store the rows of a finished aligned column.
template <class L, int W>
__device__ __forceinline__ void lut_store(const uint32_t (&f)[W][L::NF], const LutShared& sh, uint32_t nrows,
                                          uint64_t off, bool ovr) {
  constexpr int R = 4 / L::H;
#pragma unroll
  for (int g = 0; g < W; ++g)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t row = g * R + r;
      if (row < nrows) put16(sh.dst[row] + off, lut_row<L>(f[g], r), ovr);
    }
}

__device__ __forceinline__ uint4 shfl_down4(const uint4& v) {
  return make_uint4(__shfl_down_sync(kFullWarp, v.x, 1), __shfl_down_sync(kFullWarp, v.y, 1),
                    __shfl_down_sync(kFullWarp, v.z, 1), __shfl_down_sync(kFullWarp, v.w, 1));
}
__device__ __forceinline__ uint4 shfl_up4(const uint4& v) {
  return make_uint4(__shfl_up_sync(kFullWarp, v.x, 1), __shfl_up_sync(kFullWarp, v.y, 1),
                    __shfl_up_sync(kFullWarp, v.z, 1), __shfl_up_sync(kFullWarp, v.w, 1));
}

// 16 bytes of a buffer of len bytes from byte off on, bytes past the end 0.
__device__ __forceinline__ uint4 load_bytes16(const uint8_t* p, uint64_t off, uint64_t len) {
  uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
  for (int b = 0; b < 16; ++b)
    if (off + b < len) w[b >> 2] |= static_cast<uint32_t>(p[off + b]) << (8 * (b & 3));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Tiles first, first + step, ... of a job: blockDim.x columns each, or the
// blocks of an unaligned job's warps. Rows off the sources' boundaries (ragged
// row lengths) have their own mode beside unaligned sources: no granules to
// splice on the way in, one lane less lost, the aligned shapes' look-ahead and
// occupancy. Over rows of the next aligned length, 4 MiB (unaligned sources'
// path -> rows' own): Gf8D RS(20,8) +21 -> +7 %, Gf16 RS(18,8) +16 -> +6 %,
// Gf16 RS(18,4) +19 -> +12 %; 256 mixed stripes, most of them ragged, 1685 ->
// 1540 us.
template <class L, int LEV, int W, int MODE>
__device__ __forceinline__ void lut_run(const LutGeom& g, const LutShared& sh, uint64_t first, uint64_t step, bool ovr,
                                        bool fp) {
  constexpr int R = 4 / L::H;
  const uint32_t k = g.k, lane = threadIdx.x & 31u;
  LutAcc<L, W> A;
  uint32_t f[W][L::NF];
  // rows of an unaligned job: lane l holds column c, lanes 1 .. write block c
  const auto store_blocks = [&](uint64_t off, bool valid) {
#pragma unroll
    for (int q = 0; q < W; ++q)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t row = q * R + r;
        if (row >= g.nrows) continue;
        const uint4 o = lut_row<L>(f[q], r);
        uint8_t* const d = sh.dst[row] + off;
        const uint32_t dl = static_cast<uint32_t>(reinterpret_cast<uint64_t>(d)) & 15u;  // one for the warp
        if (dl == 0) {
          if (valid) put16(d, o, ovr);
        } else {
          const uint4 b = splice16(shfl_up4(o), o, 16u - dl);
          if (valid) put16(d - dl, b, ovr);
        }
      }
  };
  if constexpr (MODE == kAligned) {
    if constexpr (kLutAhead<L, W>) {
      const uint64_t end = g.head + 16 * g.ncol, stride = 16 * step * blockDim.x;
      uint64_t off = g.head + 16 * (first * blockDim.x + threadIdx.x);
      if (off >= end) return;
      LutAhead h;
#pragma unroll
      for (uint32_t j = 0; j < 3; ++j) h.c[j] = j < k ? ldg16(sh.src[j] + off) : make_uint4(0, 0, 0, 0);
      for (;;) {
        const uint64_t noff = off + stride;
        const bool more = noff < end;
        lut_column_ahead<L, W>(
            A, k, h, [&](uint32_t t) { return ldg16(sh.src[t] + off); },
            [&](uint32_t t) { return more ? ldg16(sh.src[t] + noff) : make_uint4(0, 0, 0, 0); }, LutAsIs());
        lut_finish<L, W, LEV>(A, f, fp);
        lut_store<L, W>(f, sh, g.nrows, off, ovr);
        if (!more) return;
        off = noff;
      }
    } else {
      const uint64_t ntiles = lut_tiles(g, MODE, blockDim.x);
      for (uint64_t tile = first; tile < ntiles; tile += step) {
        const uint64_t v = tile * blockDim.x + threadIdx.x;
        if (v >= g.ncol) return;
        const uint64_t o = g.head + 16 * v;
        lut_column<L, W>(A, g.k, [&](uint32_t t) { return ldg16(sh.src[t] + o); }, LutAsIs());
        lut_finish<L, W, LEV>(A, f, fp);
        lut_store<L, W>(f, sh, g.nrows, o, ovr);
      }
    }
  } else if constexpr (MODE == kRowsOff) {
    const uint32_t warps = blockDim.x >> 5;
    const uint64_t stride = step * warps * lut_warp_blocks(MODE);
    uint64_t v = lut_first_block(MODE) + (first * warps + (threadIdx.x >> 5)) * lut_warp_blocks(MODE);  // lane 1's
    // lanes past the last column read it again
    const auto column = [&](uint64_t c) { return g.head + 16 * (c < g.ncol ? c : g.ncol - 1); };
    if constexpr (kLutAhead<L, W>) {
      if (v >= g.ncol) return;
      LutAhead h;
      uint64_t off = column(v - 1 + lane);
#pragma unroll
      for (uint32_t j = 0; j < 3; ++j) h.c[j] = j < k ? ldg16(sh.src[j] + off) : make_uint4(0, 0, 0, 0);
      for (;;) {
        const uint64_t nv = v + stride, noff = column(nv - 1 + lane);
        const bool more = nv < g.ncol;
        lut_column_ahead<L, W>(
            A, k, h, [&](uint32_t t) { return ldg16(sh.src[t] + off); },
            [&](uint32_t t) { return more ? ldg16(sh.src[t] + noff) : make_uint4(0, 0, 0, 0); }, LutAsIs());
        lut_finish<L, W, LEV>(A, f, fp);
        store_blocks(off, lane >= 1 && v - 1 + lane < g.ncol);
        if (!more) return;
        v = nv;
        off = noff;
      }
    } else {
      for (; v < g.ncol; v += stride) {
        const uint64_t off = column(v - 1 + lane);
        lut_column<L, W>(A, k, [&](uint32_t t) { return ldg16(sh.src[t] + off); }, LutAsIs());
        lut_finish<L, W, LEV>(A, f, fp);
        store_blocks(off, lane >= 1 && v - 1 + lane < g.ncol);
      }
    }
  } else if (g.bytes) {  // each thread reads and writes only its own column
    for (uint64_t off = 16 * (first * blockDim.x + threadIdx.x); off < g.len; off += 16 * step * blockDim.x) {
      lut_column<L, W>(A, k, [&](uint32_t t) { return load_bytes16(sh.src[t], off, g.len); }, LutAsIs());
      lut_finish<L, W, LEV>(A, f, fp);
      const uint32_t nb = g.len - off < 16 ? static_cast<uint32_t>(g.len - off) : 16u;
#pragma unroll
      for (int q = 0; q < W; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (static_cast<uint32_t>(q * R + r) < g.nrows)
            put_bytes(sh.dst[q * R + r] + off, lut_row<L>(f[q], r), 0, nb, ovr);
    }
  } else {
    const uint32_t warps = blockDim.x >> 5;
    const uint64_t end = lut_end_block(MODE, g.ncol), stride = step * warps * lut_warp_blocks(MODE);
    uint64_t v = lut_first_block(MODE) + (first * warps + (threadIdx.x >> 5)) * lut_warp_blocks(MODE);
    for (; v < end; v += stride) {
      const uint64_t c = v - 1 + lane;
      // A granule past the last whole one belongs to no column that is written.
      lut_column<L, W>(
          A, k,
          [&](uint32_t t) {
            const uint64_t a = reinterpret_cast<uint64_t>(sh.src[t]);
            const uint32_t s = static_cast<uint32_t>(a) & 15u;
            uint4 x = make_uint4(0, 0, 0, 0);
            if (16 * c + 16 - s <= g.len) x = ldg16(reinterpret_cast<const uint8_t*>(a - s) + 16 * c);
            return x;
          },
          [&](uint32_t t, const uint4& x) {
            const uint32_t s = static_cast<uint32_t>(reinterpret_cast<uint64_t>(sh.src[t])) & 15u;  // one for the warp
            return s == 0 ? x : splice16(x, shfl_down4(x), s);
          });
      lut_finish<L, W, LEV>(A, f, fp);
      store_blocks(16 * c, lane >= 1 && lane <= lut_warp_blocks(MODE) && c < end);
    }
  }
}

// Start of edge column j of a job, its bytes (0 = none).
__device__ __forceinline__ uint64_t lut_edge(const LutGeom& g, int mode, uint32_t j, uint32_t* nb) {
  const uint64_t tail = g.head + 16 * g.ncol;
  uint64_t st = 0, n = 0;
  if (mode == kAnyOff) {
    // columns 0, 1 and ncol - 2, ncol - 1, ncol, each once
    const uint64_t lo = g.ncol >= 4 ? g.ncol - 2 : 2;
    st = 16 * (j < 2 ? j : lo + (j - 2));
    n = st < g.len ? g.len - st : 0;
    if (n > 16) n = 16;
  } else if (j == 0) {
    n = g.head;
  } else if (j == 1) {
    st = tail;
    n = g.len - tail;
  } else if (mode == kRowsOff && g.ncol >= j - 1 && j < 4) {  // the first and the last column
    st = j == 2 ? g.head : tail - 16;
    n = 16;
  }
  *nb = static_cast<uint32_t>(n);
  return st;
}

// The edge columns of a job, by one CTA: a thread stages a source's column with
// 16 independent byte loads, one thread folds a column, a thread writes a
// row's column. `stage` holds (g.k + kLutRows) * kEdges * 16 bytes.
template <class L, int LEV, int W, int MODE>
__device__ __forceinline__ void lut_edges(const LutGeom& g, const LutShared& sh, uint8_t* stage, bool ovr, bool fp) {
  constexpr int R = 4 / L::H;
  for (uint32_t i = threadIdx.x; i < g.k * kEdges; i += blockDim.x) {
    uint32_t nb;
    const uint64_t st = lut_edge(g, MODE, i % kEdges, &nb);
    reinterpret_cast<uint4*>(stage)[i] = load_bytes16(sh.src[i / kEdges] + st, 0, nb);
  }
  __syncthreads();
  uint8_t* const out = stage + g.k * kEdges * 16u;  // [row][edge][16]
  if (threadIdx.x < kEdges) {
    const uint32_t j = threadIdx.x;
    uint32_t nb;
    lut_edge(g, MODE, j, &nb);
    if (nb) {
      LutAcc<L, W> A;
      uint32_t f[W][L::NF];
      lut_column<L, W>(A, g.k, [&](uint32_t t) { return reinterpret_cast<const uint4*>(stage)[t * kEdges + j]; },
                       LutAsIs());
      lut_finish<L, W, LEV>(A, f, fp);
#pragma unroll
      for (int q = 0; q < W; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (static_cast<uint32_t>(q * R + r) < g.nrows)
            reinterpret_cast<uint4*>(out)[(q * R + r) * kEdges + j] = lut_row<L>(f[q], r);
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < g.nrows * kEdges; i += blockDim.x) {
    uint32_t nb;
    const uint64_t st = lut_edge(g, MODE, i % kEdges, &nb);
    uint8_t* const d = sh.dst[i / kEdges];
    uint32_t b0 = 0, b1 = nb;
    if (MODE != kAligned && lut_blocks(MODE, g.ncol)) {
      // the vector path wrote [w0, w1): no column reaches past both ends
      const uint32_t dl = static_cast<uint32_t>(reinterpret_cast<uint64_t>(d) + g.head) & 15u;
      const uint64_t w0 = g.head + 16 * lut_first_block(MODE) - dl, w1 = g.head + 16 * lut_end_block(MODE, g.ncol) - dl;
      if (st >= w0 && st < w1)
        b0 = w1 - st < nb ? static_cast<uint32_t>(w1 - st) : nb;
      else if (st < w0 && w0 - st < nb)
        b1 = static_cast<uint32_t>(w0 - st);
    }
    uint4 o = reinterpret_cast<const uint4*>(out)[i];
    if (!ovr && b0 < b1) {
      const uint4 x = load_bytes16(d + st, 0, nb);
      o.x ^= x.x, o.y ^= x.y, o.z ^= x.z, o.w ^= x.w;
    }
    if (b0 < b1) put_bytes(d + st + b0, o, b0, b1, true);
  }
}

}  // namespace fgfc
