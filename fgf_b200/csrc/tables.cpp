// tables.cpp -- host derivation of the product tables and images a launch uploads.
#include <algorithm>
#include <cstring>

#include "internal.hpp"

namespace fgfc {

const Gf8Log& gf8b_tab() {
  static const Gf8Log t(0x1B, 0x03);
  return t;
}
const Gf8Log& gf8d_tab() {
  static const Gf8Log t(0x1D, 0x02);
  return t;
}

Fp8Log::Fp8Log() {
  uint8_t v = 1;
  for (int i = 0; i < 255; ++i) {
    exp[i] = exp[i + 255] = v;
    log[v] = static_cast<uint8_t>(i);
    v = static_cast<uint8_t>(fp_mul_bits(v, 0x2D, 8));
  }
  exp[510] = exp[511] = 1;
  log[0] = 0;
}
const Fp8Log& fp8_tab() {
  static const Fp8Log t;
  return t;
}

namespace {

// Logarithm tables of a field of bytes.
struct ByteLogs {
  const uint8_t *exp, *log;
};
ByteLogs byte_logs(int field) {
  if (field == kFp8) return {fp8_tab().exp, fp8_tab().log};
  const Gf8Log& t = field == kGf8D ? gf8d_tab() : gf8b_tab();
  return {t.exp, t.log};
}

}  // namespace

void build_compact_tables(int field, const uint64_t* coeffs, size_t m, size_t k, uint32_t* out) {
  const ByteLogs logs = byte_logs(field);
  for (size_t t = 0; t < k; ++t) {
    uint32_t bit[8] = {0};  // products by each input bit, byte j of row j
    for (size_t j = 0; j < m; ++j)
      if (const uint8_t c = static_cast<uint8_t>(coeffs[t * m + j]))
        for (int b = 0; b < 8; ++b) bit[b] |= static_cast<uint32_t>(logs.exp[logs.log[c] + logs.log[1 << b]]) << (8 * j);
    uint32_t* w = out + t * kCompactWords;
    for (int half = 0; half < 2; ++half, w += 16) {
      w[0] = 0;
      for (uint32_t n = 1; n < 16; ++n) {  // the lowest set bit and the rest
        const int low = n & 1 ? 0 : n & 2 ? 1 : n & 4 ? 2 : 3;
        w[n] = w[n & (n - 1)] ^ bit[4 * half + low];
      }
    }
  }
}

// Tower levels split per launch. A leaf product's table word holds the H-byte
// products of 4 / H rows, and an element takes 8 H / 5 lookups per leaf product
// and word, so (lookups per element, source and word set, in input bytes):
//   2 bytes: direct 2 per 2 rows, halves 3 per 4 rows;
//   4 bytes: direct 4 per row, 16-bit leaves 6 per 2 rows, byte leaves 9 per 4;
//   8 bytes: 32-bit leaves 12 per row, 16-bit 18 per 2 rows, byte leaves 27 per 4.
// The splits cost a fix-up per column whatever the number of sources, so the 2-
// and 4-byte fields go direct, a word per 4 / E rows, with one source, and with
// two unless the rows fill a split's words. 16 MiB, us, split -> direct: Gf32 k = 1,
// m = 3 34.5 -> 19.8, m = 8 added 114 -> 78; k = 2, m = 3 43.0 -> 32.5, m = 4 44.6
// -> 39.8 but 5.0 -> 6.1 at 64 KiB; Gf16 k = 1, m = 4 21.7 -> 16.2.
LutShape lut_shape(int E, size_t nr, size_t k) {
  LutShape s{};
  if (E == 1) {
    s.w = static_cast<int>((nr + 3) / 4);
  } else if (E <= 4 && (k == 1 || (k == 2 && nr * E < 16))) {
    s.w = static_cast<int>((nr * E + 3) / 4);
  } else if (E == 2) {
    s.lev = nr > 2 ? 1 : 0;
    s.w = nr > 4 ? 2 : 1;
  } else if (E == 4) {
    s.lev = nr > 2 ? 2 : nr > 1 ? 1 : 0;
    s.w = 1;
  } else {
    s.lev = nr > 2 ? 3 : nr > 1 ? 2 : 1;
    s.w = 1;
  }
  s.nv = static_cast<size_t>(E >> s.lev);
  for (int i = 0; i < s.lev; ++i) s.nv *= 3;
  return s;
}

size_t lut_sources(const LutShape& s, bool inl) {
  const size_t edge = kEdges * 16;  // staged edge columns per source and row
  size_t kc = std::min<size_t>(kMaxSrc, (kLutSmemMax - kLutRows * edge) / (s.smem3() + 3 * edge) * 3);
  if (inl) kc = std::min<size_t>(kc, kLutInlineWords / s.src_words());
  return kc;
}

size_t lut_image_words(int E, size_t k, size_t m) {
  size_t n = 0;
  for (size_t r0 = 0; r0 < m; r0 += lut_rows(E)) n += k * lut_shape(E, std::min(lut_rows(E), m - r0), k).src_words();
  return n;
}

namespace {

// The field one level's leaves live in: `field`'s subfield of H bytes.
int leaf_field(int field, int H) {
  if (field == kFp8 || field == kFp16 || field == kFp32 || field == kFp64)
    return H == 1 ? kFp8 : H == 2 ? kFp16 : H == 4 ? kFp32 : kFp64;
  if (field == kGf8D) return kGf8D;
  return H == 1 ? kGf8B : H == 2 ? kGf16 : H == 4 ? kGf32 : kGf64;
}

}  // namespace

void build_lut_images(int field, const LutShape& shape, const uint64_t* coeffs, size_t m, size_t t0, size_t k, size_t r0,
                      size_t nr, uint32_t* out) {
  const int E = field_bytes(field), lev = shape.lev;
  const int H = E >> lev, leaf = leaf_field(field, H);
  const ByteLogs byte = byte_logs(leaf_field(field, 1));
  int two[8];  // logarithms of a byte's bits
  for (int b = 0; b < 8; ++b) two[b] = byte.log[1 << b];
  const size_t W = static_cast<size_t>(shape.w), nv = shape.nv;
  std::memset(out, 0, k * shape.src_words() * sizeof(uint32_t));
  for (size_t t = 0; t < k; ++t)
    for (size_t r = 0; r < nr; ++r) {
      // v[P][i]: product P by bit i. The element's leaves are multiplied by each
      // byte's 1, bytes scale the others (the byte level is a subfield), and the
      // products of sums of leaves are sums of theirs.
      uint32_t v[27][32];
      const uint64_t c = coeffs[(t0 + t) * m + r0 + r] & field_mask(field);
      int at[8], n = 1 << lev;  // where each leaf's product stands in tree order
      for (int l = 0; l < n; ++l) {
        at[l] = 0;
        for (int d = lev; d-- > 0;) at[l] = 3 * at[l] + (l >> d & 1);
        const uint64_t cl = c >> (8 * H * l) & field_mask(leaf);
        for (int p = 0; p < H; ++p) {
          const uint64_t one = p ? gf_mul(leaf, cl, 1ull << (8 * p)) : cl;
          uint32_t* x = v[at[l]] + 8 * p;
          for (int b = 0; b < 8; ++b) x[b] = 0;
          for (int o = 0; o < H; ++o)
            if (const uint8_t a = static_cast<uint8_t>(one >> (8 * o)))
              for (int b = 0; b < 8; ++b) x[b] |= static_cast<uint32_t>(byte.exp[byte.log[a] + two[b]]) << (8 * o);
        }
      }
      for (int sub = 1; sub < static_cast<int>(nv) / H; sub *= 3)  // products below a split: low, high, their sum
        for (int P = 0; P < static_cast<int>(nv) / H; ++P)
          if (P / sub % 3 == 2)
            for (int i = 0; i < 8 * H; ++i) v[P][i] = v[P - 2 * sub][i] ^ v[P - sub][i];
      for (size_t P = 0; P < nv / H; ++P)
        for (int i = 0; i < 8 * H; ++i)
          for (int o = 0; o < H; ++o) {
            const size_t f = r * H + o;  // output byte: word f / 4
            out[((t * nv + P * H + i / 8) * W + f / 4) * 8 + i % 8] |= (v[P][i] >> (8 * o) & 0xFFu) << (8 * (f % 4));
          }
    }
}

cudaError_t lut_launch(int field, const LutShape& sh, LutArgs& a, int mode, cudaStream_t s) {
  const int E = field_bytes(field);
  a.fp = field == kFp16 || field == kFp32 || field == kFp64 ? 1u : 0u;
  switch (E) {
    case 1: return lut_launch_e1(sh.lev, sh.w, a, s, mode);
    case 2: return lut_launch_e2(sh.lev, sh.w, a, s, mode);
    case 4: return lut_launch_e4(sh.lev, sh.w, a, s, mode);
    case 8: return lut_launch_e8(sh.lev, sh.w, a, s, mode);
    default: return cudaErrorInvalidValue;
  }
}

LutBatchKernel lut_batch_kernel_for(int E, LutShape s, int mode) {
  switch (E) {
    case 1: return lut_batch_e1(s.lev, s.w, mode);
    case 2: return lut_batch_e2(s.lev, s.w, mode);
    case 4: return lut_batch_e4(s.lev, s.w, mode);
    case 8: return lut_batch_e8(s.lev, s.w, mode);
    default: return LutBatchKernel{};
  }
}

JobAlign job_align(int field, const uint64_t* srcs, size_t k, const uint64_t* dsts, size_t m, uint64_t len) {
  JobAlign r{true, false, false, 0, kAligned};
  const uint64_t al = k ? srcs[0] & 15 : 0;
  for (size_t t = 0; t < k; ++t) r.sources = r.sources && (srcs[t] & 15) == al;
  r.sources = r.sources && al % static_cast<uint64_t>(field_bytes(field)) == 0;
  r.unal = !r.sources;
  for (size_t j = 0; j < m; ++j) r.unal = r.unal || (dsts[j] & 15) != al;
  if (r.unal)
    for (size_t j = 0; j < m; ++j)
      for (size_t t = 0; t < k; ++t) r.overlap = r.overlap || (dsts[j] < srcs[t] + len && srcs[t] < dsts[j] + len);
  if (r.sources) r.head = std::min<uint64_t>((16 - al) & 15, len);
  r.mode = !r.unal ? kAligned : r.sources && !r.overlap ? kRowsOff : kAnyOff;
  return r;
}

}  // namespace fgfc
