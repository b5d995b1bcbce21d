// Shared host/device helpers of the es_b200 library (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include <nvtx3/nvToolsExt.h>

#include "es_b200.h"

namespace es_b200 {

// ---- host: error reporting ------------------------------------------------------------------
char* last_error_buffer();            // thread-local, 512 bytes
int fail(int code, const char* fmt, ...);

#define ES_CUDA_TRY(expr)                                                                   \
  do {                                                                                      \
    cudaError_t _e = (expr);                                                                \
    if (_e != cudaSuccess)                                                                  \
      return ::es_b200::fail(ES_B200_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(_e)); \
  } while (0)

#define ES_REQUIRE(cond, ...)                                                        \
  do {                                                                               \
    if (!(cond)) return ::es_b200::fail(ES_B200_ERR_INVALID_ARGUMENT, __VA_ARGS__);  \
  } while (0)

// Cached per-device properties (SM count, compute capability).  Queried once per device.
struct DeviceInfo {
  int sm_count;
  int cc_major;
  int cc_minor;
};
int get_device_info(DeviceInfo* out);   // for the current device

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ---- host: NVTX range around the launches of one operator call ---------------------------------
// (header-only NVTX: a no-op unless a profiler is attached; makes a tool's launch list attributable per operator, as the
// reference's benchmark does around its call: benchmark_sm100_mxfp8_blockscaled_moe.py:112-114)
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

// ---- host: tunables ----------------------------------------------------------------------------
// One set per process; each has a built-in default, an environment override read once (ES_B200_<NAME in capitals>)
// and can be changed at run time with es_b200_set_tunable.
struct Tunables {
  int mm_heavy_min_rows;        // MXFP8 GEMM: experts with at least this many rows are the heavy ones of the work list; 0 = built-in
  int mm_pair_max_clusters;     // cap of the grid in CTA pairs (0 = as many as fit)
  int mm_dynamic;               // 1: items are dealt through the work counters in scratch when scratch is given
  int mm_item_k_steps;          // a work item spans enough weight pairs for this many K steps (<= 8 pairs)
  // names of earlier versions (several kernels per call); accepted, without effect
  int mm_tiny_max_rows, mm_pair_first_clusters, mm_split_min_rows, mm_stream_max_ctas, mm_stream_lsu, mm_stream_mid_lead_ctas;
};
Tunables& tunables();
void note_device_error();   // es_b200_check_status found status bits set (see es_b200_error_epoch)

// ---- device: programmatic dependent launch ---------------------------------------------------
// Both are no-ops when the kernel was not launched with the programmatic-stream-serialization attribute.
__device__ __forceinline__ void pdl_wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- work counters of the MXFP8 grouped GEMM ---------------------------------------------------
// The scratch of a call holds two 32-bit words, zero between calls: [0] items dealt so far (beyond the first one of every CTA
// pair), [1] CTAs that are done.  The last CTA of the call clears both.
constexpr size_t GROUPED_MM_SCRATCH_BYTES = 256;
constexpr uint32_t ERR_SCALE_OFFSET_BIT = 0x80u;   // a blockscale offset that is not a multiple of 128 rows

// ---- device: block-wide exclusive scan of up to 1024 per-expert counts -----------------------
// counts are produced by `f(e)` for e in [0, n); results go to prefix[0..n] (prefix[n] = total).
// Must be called by all threads of a block whose size is a multiple of 32 and at most 1024.
template <class F>
__device__ __forceinline__ void block_exclusive_scan(int n, int* prefix, int* warp_sums /*[32]*/, F f) {
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  const int per = (n + nthr - 1) / nthr;      // consecutive experts per thread
  const int lo = tid * per;
  int local = 0;
  for (int i = 0; i < per; ++i) {
    int e = lo + i;
    if (e < n) local += f(e);
  }
  // inclusive warp scan of `local`
  const int lane = tid & 31, warp = tid >> 5;
  int incl = local;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int nw = nthr >> 5;
    int v = lane < nw ? warp_sums[lane] : 0;
    int s = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= d) s += t;
    }
    warp_sums[lane] = s - v;   // exclusive
  }
  __syncthreads();
  int run = warp_sums[warp] + incl - local;
  for (int i = 0; i < per; ++i) {
    int e = lo + i;
    if (e < n) {
      prefix[e] = run;
      run += f(e);
    }
  }
  if (tid == nthr - 1) prefix[n] = run;   // last thread holds the grand total (threads past n add 0)
  __syncthreads();
}

// largest e in [0, n) with prefix[e] <= u  (prefix non-decreasing, prefix[0] = 0, u < prefix[n])
__device__ __forceinline__ int upper_bound_expert(const int* prefix, int n, int u) {
  int lo = 0, hi = n;   // invariant: prefix[lo] <= u < prefix[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (prefix[mid] <= u) lo = mid; else hi = mid;
  }
  return lo;
}

// ---- device: per-expert facts in shared memory ------------------------------------------------
// Every role of a grouped GEMM kernel needs the expert's row count, first row and first scale row for every work
// item.  Read from global memory that is a chain of dependent L2 round trips per item (~2000 cycles behind the binary
// search over the item prefix), which an MMA-issuing lane cannot hide when an item has only a few K steps.  The
// kernels therefore copy them once per CTA into the tail of the array that holds the item prefix: `table` has
// ES_B200_MAX_EXPERTS + 1 ints, the prefix takes n + 1 of them, the copies of as many experts as fit follow (all of
// them when n <= 256 with three tables); experts beyond that are read from global memory as before.
struct ExpertTable {
  const int* prefix;
  const int* rows;              // shared-memory copies for experts below `cached`
  const int* first_row;
  const int* scale_row0;
  int cached;
  const int* problem_sizes;     // global memory
  const int* expert_offsets;
  const int* blockscale_offsets;   // may be null (no third table)
  __device__ __forceinline__ int m(int e) const { return e < cached ? rows[e] : problem_sizes[e * 3]; }
  __device__ __forceinline__ int row0(int e) const { return e < cached ? first_row[e] : expert_offsets[e]; }
  __device__ __forceinline__ int scale0(int e) const { return e < cached ? scale_row0[e] : blockscale_offsets[e]; }
};
// Called by all threads after block_exclusive_scan has written table[0..n]; the caller synchronises the block before
// the table is read.
__device__ __forceinline__ ExpertTable fill_expert_table(int* table, int n, const int* problem_sizes,
                                                         const int* expert_offsets, const int* blockscale_offsets) {
  ExpertTable tab;
  const int tables = blockscale_offsets ? 3 : 2;
  const int room = (ES_B200_MAX_EXPERTS + 1 - (n + 1)) / tables;
  tab.cached = n < room ? n : room;
  int* rows = table + n + 1;
  int* first_row = rows + tab.cached;
  int* scale_row0 = first_row + tab.cached;
  for (int e = threadIdx.x; e < tab.cached; e += blockDim.x) {
    rows[e] = problem_sizes[e * 3];
    first_row[e] = expert_offsets[e];
    if (blockscale_offsets) scale_row0[e] = blockscale_offsets[e];
  }
  tab.prefix = table;
  tab.rows = rows;
  tab.first_row = first_row;
  tab.scale_row0 = scale_row0;
  tab.problem_sizes = problem_sizes;
  tab.expert_offsets = expert_offsets;
  tab.blockscale_offsets = blockscale_offsets;
  return tab;
}

}  // namespace es_b200
