// internal.hpp -- shared declarations between the C ABI layer (api.cpp) and
// the device code (kernels.cu) of libfgfcuda.so.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

#include "../../include/fgf_cuda.h"
#include "gf_host.hpp"

namespace fgfc {

// Limits of one kernel launch. Calls with more sources or rows are split
// into several launches by the host (exact: rows are independent, and
// sources split into an overwrite launch followed by accumulate launches).
constexpr int kMaxSrc = 64;
constexpr size_t kFastMaxSources = 14;   // byte-table kernels: sources per launch
// Their compact tables, per source: word[n] (n < 16) = products of the low
// nibble value n, word[16 + n] = products of n << 4; byte q is row q.
constexpr int kCompactWords = 32;

struct MatrixLaunch {
  uint64_t len;            // bytes per row
  uint64_t head;           // bytes before the vector body
  uint64_t nvec;           // 16-byte vectors in the body
  uint32_t k;              // sources
  uint32_t nrows;          // rows written by this launch (<= 4)
  uint32_t shift;          // 1: some row is not at the sources' offset within 16 bytes
  const uint32_t* tables;  // device compact tables, or nullptr for `inline_tab`
  const uint8_t* src[kFastMaxSources];
  uint8_t* dst[4];
  uint32_t inline_tab[kFastMaxSources * kCompactWords];
};

// Compact tables of a term-major k x m (m <= 4) matrix over a 1-byte field.
void build_compact_tables(int field, const uint64_t* coeffs, size_t m, size_t k, uint32_t* out);

// ---------------------------------------------------------------- table kernels (lut.cuh)

// How a job's pointers sit within 16 bytes.
enum LutMode : int {
  kAligned = 0,  // every source and row at one offset, whole elements before the boundary
  kRowsOff = 1,  // the sources so, rows anywhere (contiguous rows of a ragged length)
  kAnyOff = 2,   // sources anywhere, or an in-place call off the boundaries
};

// One job's geometry. Columns are 16 bytes, column v at head + 16 v: the first
// boundary of the sources, or the row's start (kAnyOff). Bytes outside the
// columns that the vector path writes are "edges".
struct LutGeom {
  uint64_t len, head, ncol;
  uint32_t k, nrows;
  uint32_t ovr;    // 1 = overwrite
  uint32_t bytes;  // kAnyOff, in place: columns are read and written bytewise
};

constexpr uint32_t kEdges = 5;  // edge columns of a job, at most
#ifdef __CUDACC__
#define FGFC_HD __host__ __device__
#else
#define FGFC_HD
#endif
// Blocks of 16 row bytes that the vector path of an unaligned job writes: block
// v ends inside column v and starts inside column v - 1, as far as the row's
// offset goes back. kRowsOff: v = 1 .. ncol - 1. kAnyOff: v = 2 .. ncol - 2 (a
// source's 16-byte granules may reach past the columns around those).
FGFC_HD constexpr uint64_t lut_first_block(int mode) { return mode == kAnyOff ? 2 : 1; }
FGFC_HD constexpr uint64_t lut_end_block(int mode, uint64_t ncol) { return mode == kAnyOff ? ncol - 1 : ncol; }
FGFC_HD constexpr uint64_t lut_blocks(int mode, uint64_t ncol) {
  return mode == kAnyOff ? (ncol >= 4 ? ncol - 3 : 0) : ncol >= 2 ? ncol - 1 : 0;
}
// Of a warp's 32 columns, lane 0's only supplies the bytes before lane 1's;
// with unaligned sources lane 31's 16 bytes only complete lane 30's.
FGFC_HD constexpr uint32_t lut_warp_blocks(int mode) { return mode == kAnyOff ? 30 : 31; }
// Does the job leave bytes to the edge pass?
FGFC_HD inline bool lut_has_edges(const LutGeom& g, int mode) {
  if (mode != kAligned) return !g.bytes;
  return g.head != 0 || g.head + 16 * g.ncol != g.len;
}
// Tiles of a job for CTAs of `threads`: a column per thread, or the blocks of
// its warps.
FGFC_HD inline uint64_t lut_tiles(const LutGeom& g, int mode, uint32_t threads) {
  if (mode == kAligned) return (g.ncol + threads - 1) / threads;
  if (g.bytes) return (g.len + 16 * threads - 1) / (16 * threads);
  const uint32_t step = threads / 32 * lut_warp_blocks(mode);
  return (lut_blocks(mode, g.ncol) + step - 1) / step;
}

constexpr int kLutThreads = 256;
constexpr int kLutRows = 16;               // rows per launch (Gf8; 8 / 4 / 4 for 2, 4 and 8 bytes)
constexpr int kLutInlineWords = 768;       // images carried in launch parameters: 3 of their 4 KiB
constexpr int kLutSmemMax = 110 * 1024;    // tables of one CTA: two CTAs per SM
struct LutArgs {
  const uint32_t* img;  // device images, or nullptr: inl
  LutGeom g;
  uint32_t fp;          // Fan-Paar fix-ups
  uint32_t edge_cta;    // 1: the last CTA takes the edges
  uint64_t ntiles;
  const uint8_t* src[kMaxSrc];
  uint8_t* dst[kLutRows];
  alignas(16) uint32_t inl[kLutInlineWords];
};
static_assert(sizeof(LutArgs) <= 4096, "launches with more than 4 KiB of parameters cost more");

// Tower levels split and output words per leaf product of a launch of nr rows
// of a call of k sources.
struct LutShape {
  int lev, w;
  size_t nv;  // leaf input bytes per element
  size_t src_words() const { return nv * static_cast<size_t>(w) * 8; }  // image words per source
  size_t smem3() const { return (nv * w * 640 + 255) / 256 * 256; }     // table bytes of three sources
  size_t smem1() const { return (nv * w * 128 + 255) / 256 * 256; }     // and of one left over
};
// Shared memory of one CTA: tables of k sources, the staged edge columns of
// the sources and of the rows.
inline uint32_t lut_smem(const LutShape& s, size_t k) {
  return static_cast<uint32_t>(k / 3 * s.smem3() + k % 3 * s.smem1() + (k + kLutRows) * kEdges * 16);
}
inline size_t lut_rows(int E) { return E == 1 ? 16 : E == 2 ? 8 : 4; }
LutShape lut_shape(int E, size_t nr, size_t k);
// Sources per launch: table pages, pointers and (raw forms) inline images fit.
size_t lut_sources(const LutShape& s, bool inl);
// Image words of k sources and m rows, launch by launch of lut_rows(E) rows.
size_t lut_image_words(int E, size_t k, size_t m);
// Images of sources [t0, t0 + k) and rows [r0, r0 + nr) of a term-major
// coefficient matrix with m columns: [source][leaf byte][word][8].
void build_lut_images(int field, const LutShape& s, const uint64_t* coeffs, size_t m, size_t t0, size_t k, size_t r0,
                      size_t nr, uint32_t* out);
// Launch one job (rows of one shape).
cudaError_t lut_launch(int field, const LutShape& sh, LutArgs& a, int mode, cudaStream_t s);
// The kernel of short rows and of few sources of the 8-byte fields (wide.cu) over
// one call: `img` holds the single-row images (build_lut_images) of coefficient
// (t, j) at (t * m + j).
bool wide_chosen(int field, size_t k, size_t m, size_t len);
// Does a batched stripe run there too, as a launch of its own?
bool wide_stripe(int field, size_t k, size_t m, size_t len);
cudaError_t wide_launch(int field, const uint8_t* const* srcs, size_t k, uint8_t* const* rows, size_t m,
                        const uint32_t* img, size_t len, bool overwrite, cudaStream_t stream);
// One descriptor of a batched submission: a byte-table sub-job (batch.cu) or a
// table sub-job (lut_batch.cuh).
struct BatchJob {
  const uint32_t* tables;  // compact tables [source][32]
  uint64_t len;            // bytes per row
  uint64_t head;           // scalar bytes before the vector body
  uint64_t nvec;           // 16-byte vectors in the body
  uint32_t k, nrows;       // sources; rows of this sub-job
  uint32_t ovr;            // 1 = overwrite
  uint32_t src_idx, dst_idx;
  uint32_t nv_items;       // vector items; scalar items follow
};
struct LutBatchJob {
  const uint32_t* img;
  LutGeom g;
  uint32_t src_idx, dst_idx;
  uint32_t parts;  // items over the tiles; one item of edges follows
  uint32_t fp;
};
union BatchDesc {
  BatchJob byte;
  LutBatchJob lut;
};
static_assert(sizeof(BatchDesc) == 64, "the no-allocation scratch limit counts 64 bytes per stripe");
using LutBatchFn = void (*)(const BatchDesc*, const uint64_t*, const void*, uint32_t, uint32_t, uint32_t*, uint32_t);
struct LutBatchKernel {
  LutBatchFn fn = nullptr;
  int ctas = 1;  // resident per SM
};
LutBatchKernel lut_batch_kernel_for(int E, LutShape s, int mode);
LutBatchKernel lut_batch_e1(int lev, int w, int mode);
LutBatchKernel lut_batch_e2(int lev, int w, int mode);
LutBatchKernel lut_batch_e4(int lev, int w, int mode);
LutBatchKernel lut_batch_e8(int lev, int w, int mode);
cudaError_t lut_launch_e1(int lev, int w, LutArgs& a, cudaStream_t s, int mode);
cudaError_t lut_launch_e2(int lev, int w, LutArgs& a, cudaStream_t s, int mode);
cudaError_t lut_launch_e4(int lev, int w, LutArgs& a, cudaStream_t s, int mode);
cudaError_t lut_launch_e8(int lev, int w, LutArgs& a, cudaStream_t s, int mode);

// The byte-table kernel (kernels.cu; Gf8, at most 4 rows, <= 14 sources); `overwrite` selects dot-product (overwrite) or
// mul_add (accumulate) semantics.
cudaError_t launch_fast_matrix(bool overwrite, const MatrixLaunch& a, cudaStream_t s);
// Fill `n` rows of `len` bytes with zero.
cudaError_t launch_zero_rows(uint8_t* const* rows, int n, uint64_t len, cudaStream_t s);
// dst ^= src over `len` bytes.
cudaError_t launch_xor(uint8_t* dst, const uint8_t* src, uint64_t len, cudaStream_t s);
// Elementwise product dst[i] = a[i] * b[i].
cudaError_t launch_elementwise(int field, uint8_t* dst, const uint8_t* a, const uint8_t* b,
                               uint64_t len, cudaStream_t s);
// The same for vectors that share their offset within 16 bytes
// (elementwise.cu): `head` bytes of whole elements, then nvec vectors of 16
// bytes, then a tail of less.
cudaError_t launch_elementwise_planes(int field, uint8_t* dst, const uint8_t* a, const uint8_t* b, uint64_t len,
                                      uint32_t head, uint64_t nvec, cudaStream_t s);

int sm_count();

// Kernel families (fgfc_kernel values) and the choice per shape (tune.cpp).
bool kernel_usable(int kernel, int field, size_t k, size_t m);
int choose_kernel(int field, size_t k, size_t m, size_t len);
// Tile shape of the batched table work lists (tune.cpp): element-vector
// columns per thread per work item for the class of element width E and G
// table groups; set_tile_cols(E, G, 0) restores the built-in value.
constexpr int kTileColsDefault = 8;
int tile_cols(int E, int G);
void set_tile_cols(int E, int G, int cols, double us);
// Shapes the bit-sliced tensor-core contraction covers in one launch
// (gf2mma.cu): at most 512 input bits and 128 output bits per element column.
bool gf2mma_shape_ok(int field, size_t k, size_t m);
// Compact GF(2) bit matrix of a term-major k x m coefficient matrix:
// kGf2BitWords words, [output bit][input word group].
constexpr size_t kGf2BitWords = 128 * 16;
void gf2mma_bits(int field, const uint64_t* coeffs, size_t k, size_t m, uint32_t* bits);
// Columns [0, nblk * 512 * E) of k sources and m rows, all 16-byte aligned.
cudaError_t gf2mma_launch(int field, const uint8_t* const* srcs, size_t k, uint8_t* const* rows, size_t m,
                          const uint32_t* bits, uint64_t nblk, bool overwrite, cudaStream_t stream);
// Several stripes of one plan in one launch: ptrs (device) holds k source and
// m row pointers per stripe, prefix (device) the first block of each stripe.
cudaError_t gf2mma_launch_multi(int field, size_t k, size_t m, const uint32_t* bits, const uint64_t* ptrs,
                                const uint64_t* prefix, uint32_t nstripes, uint64_t nblk, bool overwrite,
                                cudaStream_t stream);
// Opt the tensor-core kernel of element width E in to its shared memory on
// the current device (done before a graph capture records a launch).
cudaError_t gf2mma_prepare(int E);
// Error word of the current device's tensor-core kernels (0 = fine);
// synchronises with the device.
int gf2mma_error(bool clear);
// Opt `fn` in to `bytes` of dynamic shared memory on the current device, once
// per (device, kernel); thread-safe.
cudaError_t ensure_smem_attr(const void* fn, int bytes);

// One lowered sub-job of a batched submission: all sources of a stripe and
// the rows of one table launch.
struct LoweredJob {
  int field;
  const uint32_t* img;       // plan images of these rows
  const uint32_t* byte_tab;  // plan byte-table tables, or nullptr (not their shape)
  uint64_t len;
  size_t k, nrows;
  bool ovr;
  std::vector<uint64_t> srcs, dsts;
};
// How the sub-job's pointers sit within 16 bytes.
struct JobAlign {
  bool sources;   // every source at one offset, whole elements before the boundary
  bool unal;      // a source or row is elsewhere
  bool overlap;   // a row shares bytes with a source
  uint64_t head;  // bytes before the sources' first boundary
  LutMode mode;
};
JobAlign job_align(int field, const uint64_t* srcs, size_t k, const uint64_t* dsts, size_t m, uint64_t len);

// One stripe's 16-byte-aligned body for the tensor-core kernel in a batch:
// its k sources and m rows already offset to the body start, nblk blocks of
// 512 element columns.
struct Gf2Job {
  int field;
  const uint32_t* bits;  // the plan's GF(2) bit matrix (host copy)
  uint64_t bits_key;     // hash of the bit matrix: stripes with equal keys share a launch
  size_t k, m;
  bool ovr;
  uint64_t nblk;
  std::vector<uint64_t> ptrs;  // k sources, then m rows
};

void* batch_state_create();
void batch_state_destroy(void* state);
void batch_state_graphs(void* state, bool on);
// The table work-list classes (element width, table groups) of the state's
// last submission.
std::vector<std::pair<int, int>> batch_state_classes(const void* state);
void batch_state_stats(const void* state, size_t* launches, size_t* items, int* replayed);
cudaError_t batch_run(void* state, const std::vector<LoweredJob>& jobs, const std::vector<Gf2Job>& tc,
                      cudaStream_t stream);
// One stripe of a plan (api.cpp) as sub-jobs for batch_run: the tensor-core
// body (when the tuner picks that kernel for the shape and every pointer
// shares one offset within 16 bytes) plus table sub-jobs for the rest.
void lower_matrix_job(const fgfc_plan* plan, const std::vector<uint64_t>& srcs, const std::vector<uint64_t>& dsts,
                      size_t row_len, bool overwrite, std::vector<LoweredJob>& out, std::vector<Gf2Job>& tc);

// Error text of the calling thread (api.cpp), for entry points defined in
// other files.
fgfc_status set_error(fgfc_status st, const char* msg);
fgfc_status clear_error();
const char* last_error_text();
fgfc_status validate_matrix_call(int field, const char* name, size_t dst_len, size_t row_len,
                                 const size_t* row_starts, size_t nrows, const fgfc_slice* srcs, size_t nsrcs,
                                 const uint32_t* coeffs, int overwrite);

// Decode rows of the code [I_k ; parity] for a survivor set and erased shards,
// term-major k x nerased (decode.cpp).
fgfc_status decode_matrix(int field, const uint32_t* parity, size_t k, size_t m, const size_t* survivors,
                          const size_t* erased, size_t nerased, uint32_t* out);

// fgfc_batch_run_noalloc's work (batch.cu): jobs already validated against
// the ops' rules; returns 0 or an fgfc_status with `msg` set.
int noalloc_run(int field, const fgfc_noalloc_job* jobs, size_t njobs, cudaStream_t stream, char* msg,
                size_t msglen);

}  // namespace fgfc
