// batch.cu -- batched submissions: many stripes of uneven field, k, m and
// shard length in one persistent launch per class, driven by a device
// work-list.
//
// A submission is lowered on the host to sub-jobs (all sources of a stripe,
// the rows of one table launch) and grouped in classes:
//   * Gf8 sub-jobs of at most 4 rows and K <= 14 sources use the byte-table
//     layout (fast_core.cuh), one class per K. When every sub-job of such a
//     class shares one plan, the CTAs load the tables once and grid-stride
//     over the flattened columns of all stripes (the stripes travel in the
//     launch parameters); otherwise each CTA takes one range of the columns.
//   * everything else runs the table kernels (lut_batch.cuh) on work items
//     (sub-job, part) claimed from a counter, one class per element width,
//     tower split, output words and alignment. Items of a stripe interleave,
//     so CTAs holding consecutive items sweep one window of memory together.
// The descriptor blob (jobs, pointers, items, counters) goes to the device in
// one copy, and a submission whose structure repeats replays a captured graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/fgf_cuda.h"
#include "fast_core.cuh"
#include "internal.hpp"

namespace fgfc {

namespace {

constexpr uint32_t kFastVecPerItem = 8 * kFastThreads;
constexpr uint32_t kFastGroupsPerItem = kFastThreads;
constexpr uint32_t kClaim = 2;  // byte-table items claimed per atomic

// ---------------------------------------------------------------- byte-table classes

// Work-list kernel for Gf8 sub-jobs of at most 4 rows and exactly K sources.
// The plan's tables stay resident across consecutive items of one plan.
template <int K, bool SHIFT>
__global__ void __launch_bounds__(kFastThreads, 1)
    batch_fast_kernel(const BatchDesc* __restrict__ jobs, const uint64_t* __restrict__ ptrs,
                      const uint2* __restrict__ items, uint32_t nitems, uint32_t* counter) {
  __shared__ uint32_t s_item;
  __shared__ const uint32_t* s_tab;
  __shared__ const uint8_t* s_src[K];
  __shared__ uint8_t* s_dst[4];
  if (threadIdx.x == 0) {
    s_tab = nullptr;
  }
  const uint32_t lane4 = (threadIdx.x & 31u) * 4u;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(counter, kClaim);
    __syncthreads();
    const uint32_t first = s_item;
    if (first >= nitems) break;
    for (uint32_t it = first; it < first + kClaim && it < nitems; ++it) {
      const uint2 wi = items[it];
      const BatchJob J = jobs[wi.x].byte;
      __syncthreads();  // the previous item is done with tables and pointers
      const bool resident = s_tab == J.tables;
      if (threadIdx.x < K) s_src[threadIdx.x] = reinterpret_cast<const uint8_t*>(ptrs[J.src_idx + threadIdx.x]);
      if (threadIdx.x < J.nrows) s_dst[threadIdx.x] = reinterpret_cast<uint8_t*>(ptrs[J.dst_idx + threadIdx.x]);
      if (!resident) {
        fill_fast<K>(J.tables, nullptr);
        if (threadIdx.x == 0) {
          s_tab = J.tables;
        }
      }
      __syncthreads();
      const bool ovr = J.ovr != 0;
      if (wi.y < J.nv_items) {
        const uint64_t step = static_cast<uint64_t>(J.nv_items) * blockDim.x;
        const uint32_t lane = threadIdx.x & 31u;
        // SHIFT: whole warps iterate together (see vector_item)
        for (uint64_t vb = static_cast<uint64_t>(wi.y) * blockDim.x + threadIdx.x - (SHIFT ? lane : 0u);
             vb < J.nvec; vb += step) {
          const uint64_t v = SHIFT ? vb + lane : vb;
          const bool valid = !SHIFT || v < J.nvec;
          const uint64_t off = J.head + (valid ? v : J.nvec - 1) * 16u;
          if (v + step < J.nvec) {  // this thread's next column: into L2 now
#pragma unroll
            for (int t = 0; t < K; ++t) prefetch_l2(s_src[t] + off + step * 16u);
          }
          uint32_t w[K][4];
#pragma unroll
          for (int t = 0; t < K; ++t) {
            const uint4 x = ldg16(s_src[t] + off);
            w[t][0] = x.x;
            w[t][1] = x.y;
            w[t][2] = x.z;
            w[t][3] = x.w;
          }
          uint32_t acc[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) acc[e] = 0;
          fast_fold<K, 4>(w, acc, lane4);
          if constexpr (SHIFT)
            store_col4_any(acc, s_dst, J.nrows, off, ovr, valid);
          else
            store_col4(acc, s_dst, J.nrows, off, ovr);
        }
      } else {
        const uint64_t gi = static_cast<uint64_t>(wi.y - J.nv_items) * kFastGroupsPerItem + threadIdx.x;
        if (gi < fast_groups(J.len, J.head, J.nvec)) {
          uint64_t off;
          const int nb = fast_group(J.len, J.head, J.nvec, gi, &off);
          fast_bytes<K>(s_src, s_dst, J.nrows, off, nb, ovr, lane4);
        }
      }
    }
  }
}

// Segmented variant for byte-table classes whose sub-jobs have their own
// plans (a batched reconstruct: one decode plan per erasure pattern). The
// class's 16-byte columns are flattened in plan order (vprefix over the
// class's sub-jobs jidx[]) and every CTA takes one contiguous range of equal
// size, in whole rows of blockDim.x columns. A CTA sweeps its range like the
// uniform kernel sweeps the whole class: the threads take consecutive
// columns, so the CTA streams through one window of each source at a time,
// and it loads pointers (and, if the plan differs, tables) only where its
// range crosses into the next sub-job -- once or twice per CTA. Short work
// items claimed from a counter (batch_fast_kernel) drain the memory pipeline
// at every item boundary instead; that kernel keeps the scalar heads and
// tails of the class.
template <int K, bool SHIFT>
__global__ void __launch_bounds__(fast_threads(K, SHIFT, true), 1)
    batch_fast_segment_kernel(const BatchDesc* __restrict__ jobs, const uint64_t* __restrict__ ptrs,
                              const uint32_t* __restrict__ jidx, const uint64_t* __restrict__ vprefix,
                              uint32_t njobs) {
  __shared__ const uint32_t* s_tab;
  __shared__ const uint8_t* s_src[K];
  __shared__ uint8_t* s_dst[4];
  const uint64_t vtotal = vprefix[njobs];
  const uint64_t rows = (vtotal + blockDim.x - 1) / blockDim.x;
  const uint64_t chunk = (rows + gridDim.x - 1) / gridDim.x * blockDim.x;
  uint64_t v0 = static_cast<uint64_t>(blockIdx.x) * chunk;
  const uint64_t v1 = v0 + chunk < vtotal ? v0 + chunk : vtotal;
  if (v0 >= v1) return;  // the whole CTA: no barrier is skipped by part of it
  // the sub-job holding column v0: the last q with vprefix[q] <= v0
  uint32_t lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (vprefix[mid] <= v0) lo = mid; else hi = mid;
  }
  uint32_t q = lo;
  if (threadIdx.x == 0) {
    s_tab = nullptr;
  }
  const uint32_t lane4 = (threadIdx.x & 31u) * 4u;
  const uint32_t lane = threadIdx.x & 31u;
  while (v0 < v1) {
    while (vprefix[q + 1] <= v0) ++q;  // sub-jobs without vectors
    const uint64_t base = vprefix[q];
    const uint64_t vend = vprefix[q + 1] < v1 ? vprefix[q + 1] : v1;
    const BatchJob J = jobs[jidx[q]].byte;
    __syncthreads();  // the previous sub-job is done with tables and pointers
    const bool resident = s_tab == J.tables;
    if (threadIdx.x < K) s_src[threadIdx.x] = reinterpret_cast<const uint8_t*>(ptrs[J.src_idx + threadIdx.x]);
    if (threadIdx.x < J.nrows) s_dst[threadIdx.x] = reinterpret_cast<uint8_t*>(ptrs[J.dst_idx + threadIdx.x]);
    if (!resident) {
      fill_fast<K>(J.tables, nullptr);
      if (threadIdx.x == 0) {
        s_tab = J.tables;
      }
    }
    __syncthreads();
    const bool ovr = J.ovr != 0;
    // SHIFT: whole warps iterate together (the row stores shuffle between
    // lanes) and lanes past the end reload the last column
    uint32_t wn[K][4];
    if constexpr (fast_pipe(K, SHIFT, true)) {
      const uint64_t u = v0 + threadIdx.x < vend ? v0 + threadIdx.x : vend - 1;
      fast_load<K>(s_src, J.head + (u - base) * 16u, wn);
    }
    for (uint64_t ub = v0 + threadIdx.x - (SHIFT ? lane : 0u); ub < vend; ub += blockDim.x) {
      const uint64_t u0 = SHIFT ? ub + lane : ub;
      const bool valid = !SHIFT || u0 < vend;
      const uint64_t u = valid ? u0 : vend - 1;
      const uint64_t off = J.head + (u - base) * 16u;
      if (!fast_pipe(K, SHIFT, true) && u + blockDim.x < vend) {  // this thread's next column: into L2 now
#pragma unroll
        for (int t = 0; t < K; ++t) prefetch_l2(s_src[t] + off + blockDim.x * 16u);
      }
      uint32_t w[K][4];
      if constexpr (fast_pipe(K, SHIFT, true)) {
#pragma unroll
        for (int t = 0; t < K; ++t)
#pragma unroll
          for (int q = 0; q < 4; ++q) w[t][q] = wn[t][q];
        if (ub + blockDim.x < vend) {
          const uint64_t un = u0 + blockDim.x < vend ? u0 + blockDim.x : vend - 1;
          fast_load<K>(s_src, J.head + (un - base) * 16u, wn);
        }
      } else {
        fast_load<K>(s_src, off, w);
      }
      uint32_t acc[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) acc[e] = 0;
      fast_fold<K, 4>(w, acc, lane4);
      if constexpr (SHIFT)
        store_col4_any(acc, s_dst, J.nrows, off, ovr, valid);
      else
        store_col4(acc, s_dst, J.nrows, off, ovr);
    }
    v0 = vend;
  }
}

// Uniform-plan variant: every sub-job of the class shares one plan, so each
// CTA loads the tables once and grid-strides over the flattened column space
// of all sub-jobs (vector columns first, then scalar groups), exactly like one
// long call. The per-stripe pointers and geometry travel in the launch
// parameters (constant bank), so the per-column job lookup is a few cached
// constant loads instead of a chain of dependent global loads; a class with
// more stripes than one parameter block holds is split into launches.
constexpr int kUniformJobs = 160;

struct UJob {
  const uint8_t* src[kFastMaxK];
  uint8_t* dst[4];
  uint64_t len, head, nvec;
  uint32_t nrows, ovr;
};

struct UniformParams {
  const uint32_t* tables;
  uint32_t njobs, pad;
  uint64_t vprefix[kUniformJobs + 1];
  uint64_t gprefix[kUniformJobs + 1];
  UJob jobs[kUniformJobs];
};
static_assert(sizeof(UniformParams) <= 32000, "launch parameter block too large");

template <int K, bool SHIFT>
__global__ void __launch_bounds__(fast_threads(K, SHIFT, true), 1)
    batch_fast_uniform_kernel(const __grid_constant__ UniformParams P) {
  fill_fast<K>(P.tables, nullptr);
  const uint32_t lane4 = (threadIdx.x & 31u) * 4u;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t vtotal = P.vprefix[P.njobs];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t j = 0, jn = 0;
  // SHIFT: whole warps iterate together (the row stores shuffle between
  // lanes; a warp may straddle two stripes) and lanes past the end reload the
  // last column
  uint32_t wn[K][4];
  if constexpr (fast_pipe(K, SHIFT, true)) {
    if (tid - (SHIFT ? lane : 0u) < vtotal) {
      const uint64_t u = tid < vtotal ? tid : vtotal - 1;
      while (u >= P.vprefix[jn + 1]) ++jn;
      fast_load<K>(P.jobs[jn].src, P.jobs[jn].head + (u - P.vprefix[jn]) * 16u, wn);
    }
  }
  for (uint64_t ub = tid - (SHIFT ? lane : 0u); ub < vtotal; ub += stride) {
    const uint64_t u0 = SHIFT ? ub + lane : ub;
    const bool valid = !SHIFT || u0 < vtotal;
    const uint64_t u = valid ? u0 : vtotal - 1;
    while (u >= P.vprefix[j + 1]) ++j;
    const UJob& J = P.jobs[j];
    const uint64_t off = J.head + (u - P.vprefix[j]) * 16u;
    uint32_t w[K][4];
    if constexpr (fast_pipe(K, SHIFT, true)) {
#pragma unroll
      for (int t = 0; t < K; ++t)
#pragma unroll
        for (int q = 0; q < 4; ++q) w[t][q] = wn[t][q];
      if (ub + stride < vtotal) {
        const uint64_t un = u0 + stride < vtotal ? u0 + stride : vtotal - 1;
        while (un >= P.vprefix[jn + 1]) ++jn;
        fast_load<K>(P.jobs[jn].src, P.jobs[jn].head + (un - P.vprefix[jn]) * 16u, wn);
      }
    } else {
      const uint64_t un = u + stride;  // this thread's next column: into L2 now
      if (un < vtotal) {
        while (un >= P.vprefix[jn + 1]) ++jn;
        const UJob& JN = P.jobs[jn];
        const uint64_t offn = JN.head + (un - P.vprefix[jn]) * 16u;
#pragma unroll
        for (int t = 0; t < K; ++t) prefetch_l2(JN.src[t] + offn);
      }
      fast_load<K>(J.src, off, w);
    }
    uint32_t acc[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = 0;
    fast_fold<K, 4>(w, acc, lane4);
    if constexpr (SHIFT)
      store_col4_any(acc, J.dst, J.nrows, off, J.ovr != 0, valid);
    else
      store_col4(acc, J.dst, J.nrows, off, J.ovr != 0);
  }
  const uint64_t gtotal = P.gprefix[P.njobs];
  j = 0;
  for (uint64_t u = tid; u < gtotal; u += stride) {
    while (u >= P.gprefix[j + 1]) ++j;
    const UJob& J = P.jobs[j];
    uint64_t off;
    const int nb = fast_group(J.len, J.head, J.nvec, u - P.gprefix[j], &off);
    fast_bytes<K>(J.src, J.dst, J.nrows, off, nb, J.ovr != 0, lane4);
  }
}

using KernelFn = void (*)(const BatchDesc*, const uint64_t*, const uint2*, uint32_t, uint32_t*);
using UniformFn = void (*)(UniformParams);
using SegmentFn = void (*)(const BatchDesc*, const uint64_t*, const uint32_t*, const uint64_t*, uint32_t);

#define FGFC_K_CASES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14)

KernelFn fast_kernel_for(int K, bool shift) {
  switch (K) {
#define FGFC_CASE(k) \
  case k: return shift ? batch_fast_kernel<k, true> : batch_fast_kernel<k, false>;
    FGFC_K_CASES(FGFC_CASE)
#undef FGFC_CASE
    default: return nullptr;
  }
}

SegmentFn segment_kernel_for(int K, bool shift) {
  switch (K) {
#define FGFC_CASE(k) \
  case k: return shift ? batch_fast_segment_kernel<k, true> : batch_fast_segment_kernel<k, false>;
    FGFC_K_CASES(FGFC_CASE)
#undef FGFC_CASE
    default: return nullptr;
  }
}

UniformFn uniform_kernel_for(int K, bool shift) {
  switch (K) {
#define FGFC_CASE(k) \
  case k: return shift ? batch_fast_uniform_kernel<k, true> : batch_fast_uniform_kernel<k, false>;
    FGFC_K_CASES(FGFC_CASE)
#undef FGFC_CASE
    default: return nullptr;
  }
}

uint32_t fast_smem(int K) {
  switch (K) {
#define FGFC_CASE(k) \
  case k: return FastLayout<k>::smem;
    FGFC_K_CASES(FGFC_CASE)
#undef FGFC_CASE
    default: return 0;
  }
}

}  // namespace

// ---------------------------------------------------------------- host side

struct BatchClass {
  int E;
  int K = 0;                   // > 0: byte-table class of Gf8 sub-jobs with K sources
  LutShape shape{};            // table class
  LutBatchKernel kern;
  size_t kc = 0;               // sources per fill
  std::vector<uint32_t> jobs;  // sub-job indices, plan order
  std::vector<uint2> items;    // byte-table class: heads and tails
  size_t nitems = 0;
  uint32_t each = 0;           // table class: items of every job, if they are equal
  size_t list_bytes() const { return each ? jobs.size() * sizeof(uint32_t) : nitems * sizeof(uint2); }
  std::vector<size_t> cuts;    // first item of each launch after the first
  std::vector<uint32_t> seg_jobs;   // byte-table class with own plans: sub-jobs with vectors, plan order
  std::vector<uint64_t> seg_prefix; // and the prefix of their vector counts (the segmented launch)
  double cost = 0;             // lookups, roughly
  bool uniform = false;        // byte-table class whose sub-jobs share one plan
  bool shift = false;          // its rows are not all at the sources' offset within 16 bytes
};

// Descriptor slots used round robin: a submission waits (on the host) only
// for the one kBatchSlots submissions before it, so that many can be queued
// on the GPU at once. With an even count, alternating submissions keep their
// own slots and replay their graphs.
constexpr int kBatchSlots = 4;

struct BatchSlot {
  uint8_t* host = nullptr;  // pinned
  uint8_t* dev = nullptr;
  size_t cap = 0;
  cudaEvent_t done = nullptr;  // the last submission out of this slot finished
  cudaEvent_t up = nullptr;    // its descriptors are on the device
  cudaGraphExec_t graph = nullptr;
  std::string key;
};

// Classes of one submission run on side streams forked from the caller's
// stream, so that small classes share the GPU instead of queueing.
constexpr int kSideStreams = 4;

struct BatchState {
  std::vector<UniformParams> uparams;
  BatchSlot slot[kBatchSlots];
  int next = 0;
  bool graphs = true;
  cudaStream_t capture = nullptr;  // records graphs, and carries the descriptor copies
  cudaStream_t side[kSideStreams] = {};
  cudaEvent_t fork = nullptr, join[kSideStreams] = {};
  size_t last_launches = 0, last_items = 0;
  int last_replayed = 0;
  std::vector<std::pair<int, int>> last_classes;  // table (E, G) classes of the last submission
  mutable std::mutex mu;
};

static cudaError_t ensure_slot(BatchSlot& s, size_t bytes) {
  if (s.cap >= bytes) return cudaSuccess;
  if (s.host) cudaFreeHost(s.host);
  if (s.dev) cudaFree(s.dev);
  s.host = nullptr;
  s.dev = nullptr;
  s.cap = 0;  // until both are there
  if (s.graph) {
    cudaGraphExecDestroy(s.graph);
    s.graph = nullptr;
  }
  s.key.clear();
  size_t cap = 1 << 16;
  while (cap < bytes) cap <<= 1;
  cudaError_t e = cudaHostAlloc(&s.host, cap, cudaHostAllocDefault);
  if (e != cudaSuccess) return e;
  e = cudaMalloc(&s.dev, cap);
  if (e != cudaSuccess) return e;
  if (!s.up) {
    e = cudaEventCreateWithFlags(&s.up, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
  }
  if (!s.done) {
    e = cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
  }
  s.cap = cap;
  return cudaSuccess;
}

void* batch_state_create() { return new BatchState(); }

void batch_state_destroy(void* p) {
  BatchState* b = static_cast<BatchState*>(p);
  if (!b) return;
  for (auto& s : b->slot) {
    if (s.done) cudaEventSynchronize(s.done);
    if (s.graph) cudaGraphExecDestroy(s.graph);
    if (s.host) cudaFreeHost(s.host);
    if (s.dev) cudaFree(s.dev);
    if (s.done) cudaEventDestroy(s.done);
    if (s.up) cudaEventDestroy(s.up);
  }
  if (b->capture) cudaStreamDestroy(b->capture);
  for (int i = 0; i < kSideStreams; ++i) {
    if (b->side[i]) cudaStreamDestroy(b->side[i]);
    if (b->join[i]) cudaEventDestroy(b->join[i]);
  }
  if (b->fork) cudaEventDestroy(b->fork);
  delete b;
}

void batch_state_graphs(void* p, bool on) { static_cast<BatchState*>(p)->graphs = on; }

std::vector<std::pair<int, int>> batch_state_classes(const void* p) {
  const BatchState* b = static_cast<const BatchState*>(p);
  std::lock_guard<std::mutex> lk(b->mu);
  std::vector<std::pair<int, int>> v = b->last_classes;
  std::sort(v.begin(), v.end());
  v.erase(std::unique(v.begin(), v.end()), v.end());
  return v;
}

void batch_state_stats(const void* p, size_t* launches, size_t* items, int* replayed) {
  const BatchState* b = static_cast<const BatchState*>(p);
  if (launches) *launches = b->last_launches;
  if (items) *items = b->last_items;
  if (replayed) *replayed = b->last_replayed;
}

static size_t align16(size_t x) { return (x + 15) & ~static_cast<size_t>(15); }

// The table sub-job of rows at `a`; parts, pointers to be filled in.
static LutBatchJob lut_batch_job(int field, const uint32_t* img, const JobAlign& a, uint64_t len, size_t k, size_t nrows,
                                 bool ovr) {
  LutBatchJob J;
  std::memset(&J, 0, sizeof J);
  J.img = img;
  J.g.len = len;
  J.g.head = a.mode == kAnyOff ? 0 : a.head;
  J.g.ncol = (len - J.g.head) / 16;
  J.g.k = static_cast<uint32_t>(k);
  J.g.nrows = static_cast<uint32_t>(nrows);
  J.g.ovr = ovr ? 1u : 0u;
  J.g.bytes = a.mode == kAnyOff && a.overlap ? 1u : 0u;
  J.fp = field == kFp16 || field == kFp32 || field == kFp64 ? 1u : 0u;
  return J;
}

cudaError_t batch_run(void* state, const std::vector<LoweredJob>& jobs, const std::vector<Gf2Job>& tc,
                      cudaStream_t stream) {
  BatchState* b = static_cast<BatchState*>(state);
  std::lock_guard<std::mutex> lk(b->mu);
  b->last_launches = b->last_items = 0;
  b->last_replayed = 0;
  b->last_classes.clear();
  if (jobs.empty() && tc.empty()) return cudaSuccess;

  // ---- device descriptors, pointer array, classes (sub-jobs in plan order)
  std::vector<BatchDesc> dj(jobs.size());
  std::vector<JobAlign> al(jobs.size());
  std::vector<uint64_t> ptrs;
  size_t nptr = 0;
  for (const LoweredJob& L : jobs) nptr += L.k + L.nrows;
  ptrs.reserve(nptr);
  std::vector<std::pair<uint32_t, uint32_t>> idx(jobs.size());  // first source and row pointer
  for (size_t i = 0; i < jobs.size(); ++i) {
    const LoweredJob& L = jobs[i];
    al[i] = job_align(L.field, L.srcs.data(), L.k, L.dsts.data(), L.nrows, L.len);
    idx[i].first = static_cast<uint32_t>(ptrs.size());
    ptrs.insert(ptrs.end(), L.srcs.begin(), L.srcs.end());
    idx[i].second = static_cast<uint32_t>(ptrs.size());
    ptrs.insert(ptrs.end(), L.dsts.begin(), L.dsts.end());
  }
  std::vector<size_t> order(jobs.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = i;
  const auto before = [&](size_t a, size_t c) { return jobs[a].img < jobs[c].img; };
  if (!std::is_sorted(order.begin(), order.end(), before)) std::stable_sort(order.begin(), order.end(), before);
  // Byte-table classes (a source count K) with fewer columns than this run the
  // table kernels instead, together with the other 1-byte sub-jobs: a 1024-thread
  // CTA with 227 KiB of tables waits for a whole SM to drain, which a mixed
  // submission's dozens of small classes did one after the other (256 mixed
  // stripes, with the order of items and launches below: 1505 -> 1463 us). One call
  // of K = 10 is level at 4 MiB rows and 16 % faster by byte tables at 8 MiB (tune.cpp).
  // A class that is alone, a plan per stripe and rows at the sources' offset, has
  // nothing to wait for: up to 10 sources the byte tables win from about 2 MiB of
  // row length on (32 stripes, 4 rows, waited for, table kernels / byte tables, us:
  // 4 MiB of K = 2 30.0 / 27.6, K = 6 38.3 / 35.0, K = 10 40.8 / 37.2, K = 14 45.1 /
  // 46.3; 64 stripes of 16 KiB, K = 10, 37.1 / 41.3, 8 of 4 KiB, K = 4, 20.1 / 29.1).
  constexpr uint64_t kByteClassCols = 8u << 16, kLoneClassCols = 2u << 16;
  std::map<size_t, uint64_t> byte_cols;
  for (size_t i = 0; i < jobs.size(); ++i)
    if (jobs[i].byte_tab && al[i].sources) byte_cols[jobs[i].k] += jobs[i].len / 16;
  bool lone = tc.empty() && !jobs.empty() && jobs[0].k <= 10, own_plans = false;
  for (size_t i = 0; i < jobs.size() && lone; ++i) {
    lone = jobs[i].byte_tab && !al[i].unal && jobs[i].k == jobs[0].k;
    own_plans = own_plans || jobs[i].byte_tab != jobs[0].byte_tab;
  }
  lone = lone && own_plans && byte_cols[jobs[0].k] >= kLoneClassCols;
  std::map<int, BatchClass> classes;
  for (size_t i : order) {
    const LoweredJob& L = jobs[i];
    const int E = field_bytes(L.field);
    const bool fast = L.byte_tab && al[i].sources && (lone || byte_cols[L.k] >= kByteClassCols);
    const LutShape shape = lut_shape(E, L.nrows, L.k);
    const int key = fast ? 1000 + 2 * static_cast<int>(L.k) + al[i].unal
                         : ((E * 4 + shape.lev) * 8 + shape.w) * 3 + al[i].mode;
    const auto at = classes.try_emplace(key);
    BatchClass& c = at.first->second;
    if (at.second) {  // what its jobs share
      c.E = E;
      if (fast) {
        c.shift = al[i].unal;
        c.K = static_cast<int>(L.k);
      } else {
        c.shape = shape;
        c.kern = lut_batch_kernel_for(E, shape, al[i].mode);
        c.kc = lut_sources(shape, false);
      }
    }
    c.jobs.push_back(static_cast<uint32_t>(i));
    BatchDesc& D = dj[i];
    if (fast) {
      BatchJob& J = D.byte;
      J.tables = L.byte_tab;
      J.len = L.len;
      J.head = al[i].head;
      J.nvec = (L.len - J.head) / 16;
      J.k = static_cast<uint32_t>(L.k);
      J.nrows = static_cast<uint32_t>(L.nrows);
      J.ovr = L.ovr ? 1u : 0u;
      J.src_idx = idx[i].first;
      J.dst_idx = idx[i].second;
      J.nv_items = 0;
    } else {
      D.lut = lut_batch_job(L.field, L.img, al[i], L.len, L.k, L.nrows, L.ovr);
      D.lut.src_idx = idx[i].first;
      D.lut.dst_idx = idx[i].second;
    }
  }
  for (auto& kv : classes) {
    BatchClass& c = kv.second;
    if (c.K == 0) {
      // Items of about equal work, two for every resident CTA, at most the tile
      // shape of the job's groups (tune.cpp: tile_cols; 8 columns per thread built
      // in; jobs of 3 and 4 groups share a class); the stripes with the most
      // sources, whose items are the longest, first. An item's start
      // (descriptors, tables, a cold pipeline) costs more than the last items'
      // imbalance: 256 mixed stripes with 16, 8, 4, 3, 2 items per CTA 1438,
      // 1384, 1343, 1332, 1320 us.
      uint64_t tile[5] = {0};  // by groups
      const auto job_tile = [&](uint32_t i) -> uint64_t {
        if (c.E == 8) return kTileColsDefault;
        const int G = static_cast<int>((jobs[i].nrows * c.E + 3) / 4);
        if (!tile[G]) {
          tile[G] = static_cast<uint64_t>(tile_cols(c.E, G));
          b->last_classes.emplace_back(c.E, G);
        }
        return tile[G];
      };
      const int mode = kv.first % 3;
      const auto more = [&](uint32_t p, uint32_t q) { return jobs[p].k > jobs[q].k; };
      if (!std::is_sorted(c.jobs.begin(), c.jobs.end(), more)) std::stable_sort(c.jobs.begin(), c.jobs.end(), more);
      uint64_t total = 0;  // tiles times sources
      for (uint32_t i : c.jobs) total += lut_tiles(dj[i].lut.g, mode, kLutThreads) * jobs[i].k;
      c.cost = static_cast<double>(total) * c.shape.nv * c.shape.w * (16 / c.E);
      const uint64_t slots = 2 * static_cast<uint64_t>(sm_count() * c.kern.ctas);
      // Stripes of one plan and of the byte tables' shape: one launch per
      // kUniformJobs stripes, as the uniform kernel needs. The work list does not;
      // such a submission counts the same launches whatever its size and alignment.
      bool one_plan = jobs[c.jobs[0]].byte_tab != nullptr;
      for (uint32_t i : c.jobs) one_plan = one_plan && jobs[i].byte_tab == jobs[c.jobs[0]].byte_tab;
      for (size_t q = 0; q < c.jobs.size(); ++q) {
        const uint32_t i = c.jobs[q];
        if (one_plan && q && q % kUniformJobs == 0) c.cuts.push_back(c.nitems);
        LutBatchJob& J = dj[i].lut;
        const uint64_t per = std::max<uint64_t>(1, std::min<uint64_t>(job_tile(i), total / (slots * jobs[i].k)));
        J.parts = static_cast<uint32_t>((lut_tiles(J.g, mode, kLutThreads) + per - 1) / per);
        const uint32_t n = J.parts + (lut_has_edges(J.g, mode) ? 1u : 0u);
        c.nitems += n;
        c.each = q == 0 || n == c.each ? n : 0;
      }
      continue;
    }
    for (uint32_t i : c.jobs) c.cost += static_cast<double>(jobs[i].len) * jobs[i].k * 1.3;  // lookups per byte
    c.uniform = true;
    for (uint32_t i : c.jobs) c.uniform = c.uniform && jobs[i].byte_tab == jobs[c.jobs[0]].byte_tab;
    if (c.uniform) continue;
    for (uint32_t i : c.jobs) {
      // vectors: the segmented launch; scalar heads and tails: work items
      BatchJob& J = dj[i].byte;
      const uint64_t ngroups = fast_groups(J.len, J.head, J.nvec);
      const uint64_t ns_items = (ngroups + kFastGroupsPerItem - 1) / kFastGroupsPerItem;
      J.nv_items = static_cast<uint32_t>((J.nvec + kFastVecPerItem - 1) / kFastVecPerItem);
      if (J.nvec) {
        if (c.seg_prefix.empty()) c.seg_prefix.push_back(0);
        c.seg_jobs.push_back(i);
        c.seg_prefix.push_back(c.seg_prefix.back() + J.nvec);
      }
      for (uint64_t p = J.nv_items; p < J.nv_items + ns_items; ++p)
        c.items.push_back(make_uint2(i, static_cast<unsigned>(p)));
    }
    c.nitems = c.items.size();
  }

  // ---- blob: jobs | ptrs | per work-list class: items, counter
  size_t off = 0;
  const size_t off_jobs = off;
  off = align16(off + dj.size() * sizeof(BatchDesc));
  const size_t off_ptrs = off;
  off = align16(off + ptrs.size() * sizeof(uint64_t));
  std::vector<std::pair<size_t, size_t>> cb;  // (items, counter) offsets
  std::vector<std::pair<size_t, size_t>> sb;  // (segment jobs, segment prefix) offsets
  for (auto& kv : classes) {
    std::pair<size_t, size_t> x{0, 0}, y{0, 0};
    if (!kv.second.uniform) {
      x.first = off;
      off = align16(off + kv.second.list_bytes());
      x.second = off;
      off = align16(off + std::max<size_t>(64, 4 * (kv.second.cuts.size() + 1)));
      if (!kv.second.seg_jobs.empty()) {
        y.first = off;
        off = align16(off + kv.second.seg_jobs.size() * sizeof(uint32_t));
        y.second = off;
        off = align16(off + kv.second.seg_prefix.size() * sizeof(uint64_t));
      }
    }
    cb.push_back(x);
    sb.push_back(y);
  }
  // tensor-core bodies: one launch per plan (bit matrix), its stripes'
  // pointers and first blocks in the blob
  struct TcGroup {
    std::vector<size_t> idx;
    size_t off_ptrs = 0, off_prefix = 0;
    uint64_t nblk = 0;
  };
  std::vector<TcGroup> tcg;
  {
    std::map<std::tuple<uint64_t, int, size_t, size_t, bool>, size_t> gi;
    for (size_t i = 0; i < tc.size(); ++i) {
      const Gf2Job& J = tc[i];
      const auto key = std::make_tuple(J.bits_key, J.field, J.k, J.m, J.ovr);
      auto it = gi.find(key);
      if (it == gi.end()) {
        it = gi.emplace(key, tcg.size()).first;
        tcg.emplace_back();
      }
      TcGroup& G = tcg[it->second];
      G.idx.push_back(i);
      G.nblk += J.nblk;
    }
    for (TcGroup& G : tcg) {
      const Gf2Job& J0 = tc[G.idx[0]];
      G.off_ptrs = off;
      off = align16(off + G.idx.size() * (J0.k + J0.m) * sizeof(uint64_t));
      G.off_prefix = off;
      off = align16(off + (G.idx.size() + 1) * sizeof(uint64_t));
    }
  }
  const size_t bytes = off;

  BatchSlot& s = b->slot[b->next];
  b->next = (b->next + 1) % kBatchSlots;
  cudaError_t e = cudaSuccess;
  if (s.done) {
    e = cudaEventSynchronize(s.done);  // the previous submission out of this slot finished
    if (e == cudaSuccess) e = cudaEventSynchronize(s.up);  // and its copy, should it have failed after that
    if (e != cudaSuccess) return e;
  }
  e = ensure_slot(s, bytes);
  if (e != cudaSuccess) return e;
  std::memcpy(s.host + off_jobs, dj.data(), dj.size() * sizeof(BatchDesc));
  std::memcpy(s.host + off_ptrs, ptrs.data(), ptrs.size() * sizeof(uint64_t));
  {
    size_t ci = 0;
    for (auto& kv : classes) {
      const auto& y = sb[ci];
      const auto& x = cb[ci++];
      if (kv.second.uniform) continue;
      uint2* at = reinterpret_cast<uint2*>(s.host + x.first);
      if (kv.second.K) {
        std::memcpy(at, kv.second.items.data(), kv.second.list_bytes());
      } else if (kv.second.each) {
        std::memcpy(at, kv.second.jobs.data(), kv.second.list_bytes());
      } else {
        for (uint32_t i : kv.second.jobs) {
          const LutBatchJob& J = dj[i].lut;
          const uint32_t n = J.parts + (lut_has_edges(J.g, kv.first % 3) ? 1u : 0u);
          for (uint32_t p = 0; p < n; ++p) *at++ = make_uint2(i, p);
        }
      }
      std::memset(s.host + x.second, 0, std::max<size_t>(64, 4 * (kv.second.cuts.size() + 1)));
      if (!kv.second.seg_jobs.empty()) {
        std::memcpy(s.host + y.first, kv.second.seg_jobs.data(), kv.second.seg_jobs.size() * sizeof(uint32_t));
        std::memcpy(s.host + y.second, kv.second.seg_prefix.data(), kv.second.seg_prefix.size() * sizeof(uint64_t));
      }
    }
    for (const TcGroup& G : tcg) {
      uint64_t* hp = reinterpret_cast<uint64_t*>(s.host + G.off_ptrs);
      uint64_t* pre = reinterpret_cast<uint64_t*>(s.host + G.off_prefix);
      uint64_t acc = 0;
      size_t n = 0;
      for (size_t i : G.idx) {
        const Gf2Job& J = tc[i];
        std::memcpy(hp, J.ptrs.data(), J.ptrs.size() * sizeof(uint64_t));
        hp += J.ptrs.size();
        pre[n++] = acc;
        acc += J.nblk;
      }
      pre[n] = acc;
    }
  }

  // ---- launches (their structure is the graph key)
  struct Launch {
    KernelFn fn = nullptr;
    LutBatchFn lfn = nullptr;
    uint32_t kc = 0;
    UniformFn ufn = nullptr;
    unsigned grid = 0, threads = 0;
    uint32_t smem = 0;
    const void* items = nullptr;
    uint32_t each = 0;
    uint32_t n = 0;
    uint32_t* counter = nullptr;
    size_t uparam = 0;
    int tc_group = -1;  // >= 0: a tensor-core launch over that group's stripes
    double cost = 0;
    std::string key;
    SegmentFn sfn = nullptr;  // segmented launch over the class's vectors
    const uint32_t* seg_jobs = nullptr;
    const uint64_t* seg_prefix = nullptr;
  };
  std::vector<Launch> launches;
  std::vector<UniformParams>& uparams = b->uparams;
  uparams.clear();
  // (off_ptrs: eight pointers weigh as much as one descriptor)
  std::string key = std::to_string(reinterpret_cast<uintptr_t>(s.dev)) + ":" + std::to_string(bytes) + ":" +
                    std::to_string(off_ptrs);
  const int sms = sm_count();
  size_t ci = 0;
  for (auto& kv : classes) {
    const BatchClass& c = kv.second;
    const auto& y = sb[ci];
    const auto& x = cb[ci++];
    const bool fast = c.K > 0;
    Launch L;
    L.cost = c.cost;
    const int akey = kv.first + (c.uniform ? 10000 : 0);
    if (c.uniform) {
      L.ufn = uniform_kernel_for(c.K, c.shift);
    } else if (fast) {
      L.fn = fast_kernel_for(c.K, c.shift);
    } else {
      L.lfn = c.kern.fn;
    }
    if (!L.fn && !L.ufn && !L.lfn) return cudaErrorInvalidValue;
    if (fast) {
      L.smem = fast_smem(c.K);
      L.threads = static_cast<unsigned>(kFastThreads);
    } else {
      L.smem = lut_smem(c.shape, std::min<size_t>(jobs[c.jobs[0]].k, c.kc));  // jobs with the most sources first
      L.threads = static_cast<unsigned>(kLutThreads);
      L.kc = static_cast<uint32_t>(c.kc);
    }
    e = ensure_smem_attr(L.ufn   ? reinterpret_cast<const void*>(L.ufn)
                         : L.lfn ? reinterpret_cast<const void*>(L.lfn)
                                 : reinterpret_cast<const void*>(L.fn),
                         L.lfn ? kLutSmemMax : static_cast<int>(L.smem));
    if (e != cudaSuccess) return e;
    if (c.uniform) {
      // one launch per block of kUniformJobs stripes
      for (size_t q0 = 0; q0 < c.jobs.size(); q0 += kUniformJobs) {
        const size_t nq = std::min<size_t>(kUniformJobs, c.jobs.size() - q0);
        uparams.emplace_back();
        UniformParams& P = uparams.back();
        std::memset(&P, 0, sizeof P);
        P.tables = dj[c.jobs[q0]].byte.tables;
        P.njobs = static_cast<uint32_t>(nq);
        for (size_t q = 0; q < nq; ++q) {
          const LoweredJob& LJ = jobs[c.jobs[q0 + q]];
          const BatchJob& J = dj[c.jobs[q0 + q]].byte;
          UJob& U = P.jobs[q];
          for (size_t t = 0; t < LJ.k; ++t) U.src[t] = reinterpret_cast<const uint8_t*>(LJ.srcs[t]);
          for (size_t rr = 0; rr < 4; ++rr) U.dst[rr] = reinterpret_cast<uint8_t*>(LJ.dsts[rr < LJ.nrows ? rr : 0]);
          U.len = J.len;
          U.head = J.head;
          U.nvec = J.nvec;
          U.nrows = static_cast<uint32_t>(LJ.nrows);
          U.ovr = LJ.ovr ? 1u : 0u;
          P.vprefix[q + 1] = P.vprefix[q] + J.nvec;
          P.gprefix[q + 1] = P.gprefix[q] + fast_groups(J.len, J.head, J.nvec);
        }
        Launch U = L;
        U.threads = static_cast<unsigned>(fast_threads(c.K, c.shift, true));
        const uint64_t want = (std::max(P.vprefix[nq], P.gprefix[nq]) + U.threads - 1) / U.threads;
        U.grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(want, sms)));
        U.uparam = uparams.size() - 1;
        // the parameter block is baked into a captured graph: hash it into the key
        // (whole words: byte by byte this took 50 us of each call)
        static_assert(sizeof(UniformParams) % 8 == 0, "hashed in 8-byte words");
        uint64_t h = 1469598103934665603ull;
        const uint64_t* pw = reinterpret_cast<const uint64_t*>(&P);
        for (size_t i = 0; i < sizeof P / 8; ++i) h = (h ^ (h >> 29) ^ pw[i]) * 1099511628211ull;
        U.key = "|u" + std::to_string(akey) + "," + std::to_string(h) + "," + std::to_string(U.grid);
        launches.push_back(U);
      }
      b->last_items += c.jobs.size();
    } else {
      if (!c.seg_jobs.empty()) {
        Launch S = L;
        S.fn = nullptr;
        S.sfn = segment_kernel_for(c.K, c.shift);
        if (!S.sfn) return cudaErrorInvalidValue;
        e = ensure_smem_attr(reinterpret_cast<const void*>(S.sfn), static_cast<int>(S.smem));
        if (e != cudaSuccess) return e;
        S.n = static_cast<uint32_t>(c.seg_jobs.size());
        S.seg_jobs = reinterpret_cast<const uint32_t*>(s.dev + y.first);
        S.seg_prefix = reinterpret_cast<const uint64_t*>(s.dev + y.second);
        S.threads = static_cast<unsigned>(fast_threads(c.K, c.shift, true));
        const uint64_t rows = (c.seg_prefix.back() + S.threads - 1) / S.threads;
        S.grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(rows, sms)));
        b->last_items += c.seg_jobs.size();
        S.key = "|s" + std::to_string(akey) + "," + std::to_string(S.n) + "," + std::to_string(S.grid);
        launches.push_back(S);
      }
      if (c.nitems) {
        for (size_t q = 0; q <= c.cuts.size(); ++q) {
          const size_t i0 = q ? c.cuts[q - 1] : 0, i1 = q < c.cuts.size() ? c.cuts[q] : c.nitems;
          L.n = static_cast<uint32_t>(i1 - i0);
          L.grid = L.lfn ? static_cast<unsigned>(std::min<uint64_t>(L.n, static_cast<uint64_t>(sms) * c.kern.ctas))
                         : static_cast<unsigned>(std::min<uint64_t>((L.n + kClaim - 1) / kClaim, sms));
          L.each = c.each;
          L.items = s.dev + x.first + (c.each ? i0 / c.each * sizeof(uint32_t) : i0 * sizeof(uint2));
          L.counter = reinterpret_cast<uint32_t*>(s.dev + x.second) + q;
          L.key = "|" + std::to_string(akey) + "," + std::to_string(L.n) + "," + std::to_string(L.each) + "," +
                 std::to_string(L.grid) + "," + std::to_string(L.smem);
          launches.push_back(L);
        }
        b->last_items += c.nitems;
      }
    }
  }
  for (size_t g = 0; g < tcg.size(); ++g) {
    const Gf2Job& J0 = tc[tcg[g].idx[0]];
    e = gf2mma_prepare(field_bytes(J0.field));  // before any capture records the launch
    if (e != cudaSuccess) return e;
    Launch L;
    L.tc_group = static_cast<int>(g);
    L.cost = 1e30;
    b->last_items += tcg[g].idx.size();
    L.key = "|g" + std::to_string(J0.bits_key) + "," + std::to_string(J0.field) + "," + std::to_string(J0.k) + "," +
           std::to_string(J0.m) + "," + std::to_string(J0.ovr) + "," + std::to_string(tcg[g].idx.size()) + "," +
           std::to_string(tcg[g].nblk);
    launches.push_back(L);
  }
  // the largest class first, so that the small ones fill the others' last waves
  std::stable_sort(launches.begin(), launches.end(), [](const Launch& p, const Launch& q) { return p.cost > q.cost; });
  for (const Launch& L : launches) key += L.key;
  const BatchDesc* djobs = reinterpret_cast<const BatchDesc*>(s.dev + off_jobs);
  const uint64_t* dptrs = reinterpret_cast<const uint64_t*>(s.dev + off_ptrs);

  const int nside = launches.size() > 1 ? static_cast<int>(std::min<size_t>(launches.size(), kSideStreams)) : 0;
  for (int i = 0; i < nside; ++i) {
    if (!b->side[i]) {
      e = cudaStreamCreateWithFlags(&b->side[i], cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->join[i], cudaEventDisableTiming);
      if (e != cudaSuccess) return e;
    }
  }
  if (nside && !b->fork) {
    e = cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
  }
  // The blob of a submission that the GPU takes longer on than the host goes up on
  // the stream that records graphs, under whatever the caller's stream still runs
  // (the slot is free: its last submission finished), and the caller's stream waits
  // for it: as a node of the graph the copy and the gaps around it cost 10 us
  // between two submissions (64 stripes of 1 MiB shards, RS(10,4): encode 192.5 ->
  // 186.9 us, rebuild 203.5 -> 199.9). The host pays 5 us for it, so the others keep
  // the node: per submission, one after another, beside / node, us: 100 Gf16 stripes
  // of 2 x 2 rows of 4 KiB 33.8 / 27.2, Gf16 (10,4) of 16 KiB 30.6 / 31.4 and 64 / 55
  // alone, 32 Gf8D (10,4) of 64 KiB 17.5 / 25.9, 7 Gf8B (11,3) of 44 KiB 12.3 / 16.9.
  // The line is where 8 us and 0.2 us a sub-job pass 13 us and the time of the bytes
  // at 1.8 TB/s. Launches that carry everything in their parameters need no blob.
  bool blob = false;
  for (const Launch& L : launches) blob = blob || !L.ufn;
  uint64_t moved = 0;
  bool wide = false;  // 8-byte fields: the GPU takes longer
  for (const LoweredJob& L : jobs) {
    moved += L.len * (L.k + L.nrows);
    wide = wide || field_bytes(L.field) == 8;
  }
  for (const Gf2Job& J : tc) moved += J.nblk * 512u * static_cast<uint64_t>(field_bytes(J.field)) * (J.k + J.m);
  const bool beside = wide || jobs.size() <= 25 || moved >= (360u << 10) * static_cast<uint64_t>(jobs.size() - 25);
  if (!beside) key += "|copy";
  if (!b->capture) {
    e = cudaStreamCreateWithFlags(&b->capture, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
  }
  if (blob && beside) {
    e = cudaMemcpyAsync(s.dev, s.host, bytes, cudaMemcpyHostToDevice, b->capture);
    if (e == cudaSuccess) e = cudaEventRecord(s.up, b->capture);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, s.up, 0);
    if (e != cudaSuccess) return e;
  }
  // with several classes, fork to the side streams (class i on stream
  // i % kSideStreams) and join back
  auto enqueue = [&](cudaStream_t st) -> cudaError_t {
    cudaError_t err = cudaSuccess;
    if (blob && !beside) err = cudaMemcpyAsync(s.dev, s.host, bytes, cudaMemcpyHostToDevice, st);
    if (err != cudaSuccess) return err;
    if (nside) {
      err = cudaEventRecord(b->fork, st);
      for (int i = 0; i < nside && err == cudaSuccess; ++i) err = cudaStreamWaitEvent(b->side[i], b->fork, 0);
      if (err != cudaSuccess) return err;
    }
    for (size_t li = 0; li < launches.size(); ++li) {
      const Launch& L = launches[li];
      cudaStream_t ls = nside ? b->side[li % nside] : st;
      if (L.tc_group >= 0) {
        const TcGroup& G = tcg[L.tc_group];
        const Gf2Job& J0 = tc[G.idx[0]];
        err = gf2mma_launch_multi(J0.field, J0.k, J0.m, J0.bits, reinterpret_cast<const uint64_t*>(s.dev + G.off_ptrs),
                                  reinterpret_cast<const uint64_t*>(s.dev + G.off_prefix),
                                  static_cast<uint32_t>(G.idx.size()), G.nblk, J0.ovr, ls);
      } else if (L.ufn) {
        L.ufn<<<L.grid, L.threads, L.smem, ls>>>(uparams[L.uparam]);
        err = cudaGetLastError();
      } else if (L.sfn) {
        L.sfn<<<L.grid, L.threads, L.smem, ls>>>(djobs, dptrs, L.seg_jobs, L.seg_prefix, L.n);
        err = cudaGetLastError();
      } else if (L.lfn) {
        L.lfn<<<L.grid, L.threads, L.smem, ls>>>(djobs, dptrs, L.items, L.each, L.n, L.counter, L.kc);
        err = cudaGetLastError();
      } else {
        L.fn<<<L.grid, L.threads, L.smem, ls>>>(djobs, dptrs, static_cast<const uint2*>(L.items), L.n, L.counter);
        err = cudaGetLastError();
      }
      if (err != cudaSuccess) return err;
    }
    for (int i = 0; i < nside && err == cudaSuccess; ++i) {
      err = cudaEventRecord(b->join[i], b->side[i]);
      if (err == cudaSuccess) err = cudaStreamWaitEvent(st, b->join[i], 0);
    }
    return err;
  };

  b->last_launches = launches.size();
  if (b->graphs) {
    if (!(s.graph && s.key == key)) {
      if (s.graph) {
        cudaGraphExecDestroy(s.graph);
        s.graph = nullptr;
      }
      cudaGraph_t g = nullptr;
      e = cudaStreamBeginCapture(b->capture, cudaStreamCaptureModeThreadLocal);
      if (e != cudaSuccess) return e;
      const cudaError_t ee = enqueue(b->capture);
      e = cudaStreamEndCapture(b->capture, &g);
      if (ee != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        return ee;
      }
      if (e != cudaSuccess) return e;
      e = cudaGraphInstantiate(&s.graph, g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) {
        s.graph = nullptr;
        return e;
      }
      s.key = key;
    } else {
      b->last_replayed = 1;
    }
    e = cudaGraphLaunch(s.graph, stream);
  } else {
    e = enqueue(stream);
  }
  if (e != cudaSuccess) return e;
  return cudaEventRecord(s.done, stream);
}

// ---------------------------------------------------------------- without allocation
//
// fgfc_batch_run_noalloc: the work-list kernels above, with every byte of
// scratch they need (descriptors, pointers, work items, the claim counters and
// the stripes' compact product tables) placed in this fixed device array
// instead of device memory allocated for the call. The host side builds the
// whole blob in a fixed host array of the same size and copies it in with one
// stream-ordered copy, so nothing is allocated on either side.
//
// The host array is pageable, so the runtime stages the copy before the call
// returns: the call may block the host until the stream reaches the copy, and
// that is also what makes it safe to refill the host array on the next call.
// (Pinning the array would make the copy truly asynchronous, but then every
// call would first have to wait on an event recorded after the previous copy.)
//
// Stripes are grouped in classes as in fgfc_batch_run: Gf8 stripes of at most
// 4 rows and at most 14 sources at one offset run the byte-table kernel for
// their source count; the rest run the table kernel of their element width,
// tower split, output words and alignment. One launch per class, in order, on
// the caller's stream. The scratch limit counts a stripe's tables and items at
// 128 bytes per (source byte, 4 output bytes) and 4096 columns or 2 KiB of
// head and tail per item; what is stored (32-byte images, fewer items) fits in
// that.

static __device__ __align__(256) uint8_t g_noalloc_scratch[FGFC_NOALLOC_SCRATCH_BYTES];
alignas(256) static uint8_t g_noalloc_host[FGFC_NOALLOC_SCRATCH_BYTES];
static std::mutex g_noalloc_mu;
constexpr int kNoallocMaxDevices = 64;
static uint8_t* g_noalloc_dev[kNoallocMaxDevices];  // device address of the array, per device

namespace {

// Class of a stripe for the scratch limit: 1..14 = byte-table kernel with that
// many sources, 100 + G = G groups of 4 output bytes.
int noalloc_class(int E, size_t nsrcs, size_t nrows) {
  const int R = 4 / E;
  const size_t G = (nrows + R - 1) / R;
  if (E == 1 && G == 1 && nsrcs >= 1 && nsrcs <= static_cast<size_t>(kFastMaxK)) return static_cast<int>(nsrcs);
  return 100 + static_cast<int>(G);
}
// A class holds stripes of any number of sources.
LutShape noalloc_shape(int E, size_t nr) { return lut_shape(E, nr, kMaxSrc); }
constexpr uint32_t kNoallocCols = 4096;   // columns per item
constexpr uint32_t kNoallocGroups = 512;  // 4-byte groups per item of the limit

}  // namespace

// Returns 0, or an fgfc_status-style code with `msg` filled in.
int noalloc_run(int field, const fgfc_noalloc_job* jobs, size_t njobs, cudaStream_t stream, char* msg,
                size_t msglen) {
  // A graph recorded from this call would replay whatever the shared host
  // and device arrays hold at replay time, not this call's descriptors.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(stream, &cap);
  if (e != cudaSuccess) {
    snprintf(msg, msglen, "batch_run_noalloc: %s", cudaGetErrorString(e));
    return FGFC_ERR_CUDA;
  }
  if (cap != cudaStreamCaptureStatusNone) {
    snprintf(msg, msglen, "batch_run_noalloc: the stream is being captured; this call cannot be recorded");
    return FGFC_ERR_ARG;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  int dev = 0;
  e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kNoallocMaxDevices) {
    snprintf(msg, msglen, "batch_run_noalloc: no usable current device");
    return FGFC_ERR_CUDA;
  }
  if (!g_noalloc_dev[dev]) {
    // The array's name is only a host-side stand-in; the kernels need its
    // device address on this device.
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      snprintf(msg, msglen, "batch_run_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return FGFC_ERR_CUDA;
    }
    g_noalloc_dev[dev] = static_cast<uint8_t*>(p);
  }
  uint8_t* const dbase = g_noalloc_dev[dev];
  const int E = field_bytes(field);
  const int R = 4 / E;

  // ---- sizes: per class its items; every stripe's tables at its own G
  constexpr int kClasses = 105;  // byte tables 1..14, table kernels 101..104
  size_t nptr = 0, ntab = 0, nlive = 0;
  size_t class_items[kClasses] = {0};
  for (size_t i = 0; i < njobs; ++i) {
    const fgfc_noalloc_job& J = jobs[i];
    if (J.nrows == 0 || J.row_len == 0 || J.nsrcs == 0) continue;
    if (J.nrows > static_cast<size_t>(4 * R) || J.nsrcs > static_cast<size_t>(kMaxSrc)) {
      snprintf(msg, msglen, "batch_run_noalloc: job %zu has %zu rows and %zu sources; at most %d rows and %d sources",
               i, J.nrows, J.nsrcs, 4 * R, kMaxSrc);
      return FGFC_ERR_LIMIT;
    }
    const size_t G = (J.nrows + R - 1) / R;
    const int cls = noalloc_class(E, J.nsrcs, J.nrows);
    const bool fast = cls < 100;
    ++nlive;
    nptr += J.nsrcs + J.nrows;
    ntab += J.nsrcs * E * G * kCompactWords;
    const uint64_t nvec = J.row_len / 16 + 1;  // upper bound before alignment is known
    const uint64_t per_vec = fast ? kFastVecPerItem : kNoallocCols;
    const uint64_t per_grp = fast ? kFastGroupsPerItem : kNoallocGroups;
    class_items[cls] += (nvec + per_vec - 1) / per_vec + (J.row_len / 4 + 2 + per_grp - 1) / per_grp + 1;
  }
  const size_t off_jobs = 0;
  const size_t off_ptrs = align16(off_jobs + nlive * sizeof(BatchDesc));
  const size_t off_tabs = align16(off_ptrs + nptr * sizeof(uint64_t));
  size_t class_off[kClasses] = {0};
  size_t off = align16(off_tabs + ntab * sizeof(uint32_t));
  for (int c = 0; c < kClasses; ++c) {
    if (!class_items[c]) continue;
    class_off[c] = off;  // items, then a 64-byte counter
    off = align16(off + class_items[c] * sizeof(uint2)) + 64;
  }
  const size_t bytes = off;
  if (bytes > FGFC_NOALLOC_SCRATCH_BYTES) {
    snprintf(msg, msglen, "batch_run_noalloc: submission needs %zu bytes of scratch, more than the %u available",
             bytes, static_cast<unsigned>(FGFC_NOALLOC_SCRATCH_BYTES));
    return FGFC_ERR_LIMIT;
  }

  // ---- blob in the host array
  BatchDesc* hj = reinterpret_cast<BatchDesc*>(g_noalloc_host + off_jobs);
  uint64_t* hp = reinterpret_cast<uint64_t*>(g_noalloc_host + off_ptrs);
  uint32_t* ht = reinterpret_cast<uint32_t*>(g_noalloc_host + off_tabs);
  size_t jn = 0, pn = 0, tn = 0;
  // Launches of a class: [0] stripes at one offset (byte-table kernel where the
  // class has it), [1] the others, whose items fill the class's list from its end.
  size_t class_n[kClasses][2] = {{0}};
  uint32_t class_smem[kClasses][2] = {{0}};
  size_t class_rows[kClasses] = {0};
  for (size_t i = 0; i < njobs; ++i) {
    const fgfc_noalloc_job& S = jobs[i];
    if (S.nrows == 0 || S.row_len == 0) continue;
    if (S.nsrcs == 0) {
      if (S.overwrite) {  // an empty sum overwrites with zero
        for (size_t j = 0; j < S.nrows; ++j) {
          e = cudaMemsetAsync(S.dst + (S.row_starts ? S.row_starts[j] : j * S.row_len), 0, S.row_len, stream);
          if (e != cudaSuccess) {
            snprintf(msg, msglen, "batch_run_noalloc: %s", cudaGetErrorString(e));
            return FGFC_ERR_CUDA;
          }
        }
      }
      continue;
    }
    const size_t G = (S.nrows + R - 1) / R;
    const int cls = noalloc_class(E, S.nsrcs, S.nrows);
    const uint32_t src_idx = static_cast<uint32_t>(pn);
    for (size_t t = 0; t < S.nsrcs; ++t) hp[pn++] = reinterpret_cast<uint64_t>(S.srcs[t].ptr);
    const uint32_t dst_idx = static_cast<uint32_t>(pn);
    for (size_t j = 0; j < S.nrows; ++j)
      hp[pn++] = reinterpret_cast<uint64_t>(S.dst + (S.row_starts ? S.row_starts[j] : j * S.row_len));
    JobAlign al = job_align(field, hp + src_idx, S.nsrcs, hp + dst_idx, S.nrows, S.row_len);
    if (al.mode == kRowsOff) al.mode = kAnyOff;  // two launches per class at most
    const int var = al.mode == kAligned ? 0 : 1;
    const bool fast = cls < 100 && !al.unal;
    uint64_t cm[kMaxSrc * 16];  // coefficients reduced to the field's width, as Plan::matrix does
    for (size_t q = 0; q < S.nsrcs * S.nrows; ++q) cm[q] = S.coeffs[q] & field_mask(field);
    const uint32_t* tables = reinterpret_cast<const uint32_t*>(dbase + off_tabs) + tn;
    uint64_t nitems;
    if (fast) {
      build_compact_tables(field, cm, S.nrows, S.nsrcs, ht + tn);
      BatchJob& J = hj[jn].byte;
      J.tables = tables;
      J.len = S.row_len;
      J.head = al.head;
      J.nvec = (S.row_len - al.head) / 16;
      J.k = static_cast<uint32_t>(S.nsrcs);
      J.nrows = static_cast<uint32_t>(S.nrows);
      J.ovr = S.overwrite ? 1u : 0u;
      J.src_idx = src_idx;
      J.dst_idx = dst_idx;
      J.nv_items = static_cast<uint32_t>((J.nvec + kFastVecPerItem - 1) / kFastVecPerItem);
      nitems = J.nv_items + (fast_groups(J.len, J.head, J.nvec) + kFastGroupsPerItem - 1) / kFastGroupsPerItem;
      class_smem[cls][var] = fast_smem(cls);
    } else {
      const LutShape shape = noalloc_shape(E, S.nrows);
      build_lut_images(field, shape, cm, S.nrows, 0, S.nsrcs, 0, S.nrows, ht + tn);
      LutBatchJob& J = hj[jn].lut;
      J = lut_batch_job(field, tables, al, S.row_len, S.nsrcs, S.nrows, S.overwrite != 0);
      J.src_idx = src_idx;
      J.dst_idx = dst_idx;
      const uint64_t per = kNoallocCols / kLutThreads;
      J.parts = static_cast<uint32_t>((lut_tiles(J.g, al.mode, kLutThreads) + per - 1) / per);
      nitems = J.parts + (lut_has_edges(J.g, al.mode) ? 1 : 0);
      class_smem[cls][var] = std::max(class_smem[cls][var],
                                      lut_smem(shape, std::min(S.nsrcs, lut_sources(shape, false))));
    }
    tn += S.nsrcs * E * G * kCompactWords;
    uint2* list = reinterpret_cast<uint2*>(g_noalloc_host + class_off[cls]);
    for (uint64_t q = 0; q < nitems; ++q) {
      const size_t at = var ? class_items[cls] - 1 - class_n[cls][1] : class_n[cls][0];
      list[at] = make_uint2(static_cast<unsigned>(jn), static_cast<unsigned>(q));
      ++class_n[cls][var];
    }
    class_rows[cls] = S.nrows;  // any of the class: they share a table shape
    ++jn;
  }
  if (jn == 0) return 0;
  for (int c = 0; c < kClasses; ++c)  // every claim counter starts at zero on every call
    if (class_items[c]) std::memset(g_noalloc_host + align16(class_off[c] + class_items[c] * sizeof(uint2)), 0, 64);

  // ---- one copy, then one launch of the work-list kernel per class
  e = cudaMemcpyAsync(dbase, g_noalloc_host, bytes, cudaMemcpyHostToDevice, stream);
  for (int c = 0; c < kClasses && e == cudaSuccess; ++c) {
    for (int var = 0; var < 2 && e == cudaSuccess; ++var) {
      const size_t n = class_n[c][var];
      if (!n) continue;
      const bool fast = c < 100 && var == 0;
      const KernelFn fn = fast ? fast_kernel_for(c, false) : nullptr;
      const LutBatchKernel lut = fast ? LutBatchKernel{} : lut_batch_kernel_for(E, noalloc_shape(E, class_rows[c]), var ? kAnyOff : kAligned);
      if (!fn && !lut.fn) {
        e = cudaErrorInvalidValue;
        break;
      }
      const uint32_t smem = class_smem[c][var];
      e = ensure_smem_attr(fast ? reinterpret_cast<const void*>(fn) : reinterpret_cast<const void*>(lut.fn),
                           fast ? static_cast<int>(smem) : kLutSmemMax);
      if (e != cudaSuccess) break;
      const BatchDesc* descs = reinterpret_cast<const BatchDesc*>(dbase + off_jobs);
      const uint64_t* ptrs = reinterpret_cast<const uint64_t*>(dbase + off_ptrs);
      const uint2* list = reinterpret_cast<const uint2*>(dbase + class_off[c]) + (var ? class_items[c] - n : 0);
      uint32_t* counter =
          reinterpret_cast<uint32_t*>(dbase + align16(class_off[c] + class_items[c] * sizeof(uint2))) + var;
      const uint64_t sms = static_cast<uint64_t>(sm_count());
      if (fast)
        fn<<<static_cast<unsigned>(std::min<uint64_t>((n + kClaim - 1) / kClaim, sms)), kFastThreads, smem, stream>>>(
            descs, ptrs, list, static_cast<uint32_t>(n), counter);
      else
        lut.fn<<<static_cast<unsigned>(std::min<uint64_t>(n, sms * lut.ctas)), kLutThreads, smem, stream>>>(
            descs, ptrs, list, 0u, static_cast<uint32_t>(n), counter,
            static_cast<uint32_t>(lut_sources(noalloc_shape(E, class_rows[c]), false)));
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) {
    snprintf(msg, msglen, "batch_run_noalloc: CUDA error: %s", cudaGetErrorString(e));
    return FGFC_ERR_CUDA;
  }
  return 0;
}

}  // namespace fgfc
