// FP8-blockwise grouped GEMM for sm_100a, experts with more than 32 token rows (see fp8_blockwise_grouped_mm.cu for the
// operator and its split into two kernels): 128 TOKEN rows on the MMA M axis, 128 weight rows (output columns) on the N
// axis, one CTA per SM.
//
// What bounds it: operand traffic.  With the promotion switched off and a quarter of the MMAs issued, 128 experts of 192
// rows at n = 768, k = 4096 take 108 us against 157 with everything on: the 1.6 GB of 16 KB tiles at 15 TB/s out of L2;
// and per K block TMA writes 32 KB of shared memory and the MMAs read as much, 512 cycles at 128 bytes per cycle for 256 of
// tensor time.  Next to that traffic every shared-memory round trip of the roles (an mbarrier wait, a broadcast read)
// takes hundreds of cycles instead of thirty: scales do not go through shared memory.  Measured on the way: 128 x 256 tiles
// (a quarter less traffic) hold 64 accumulators a thread, spill, and were 14 % slower; two K blocks per stage and
// hand-over 13 % slower; the kernel serving the experts of <= 32 rows too (128 MMA rows for a few tokens) 4-8 % slower
// there than the few-rows kernel.
// Two K blocks share a barrier round trip between the MMA thread and the promotion, whose TMEM reads overlap its
// multiplications: with one K block per round trip and no overlap the promotion set the pace (780 cycles per K block; 585
// now, of which 512 are the shared-memory pipe's), 165 us against 155.  The whole call took 212 with the tokens on N.  Experts of
// 33 to 64 rows, whose MMAs are half empty, gain as well, at long K too (bound by HBM): E = 256, 48 rows, n = 512, k = 7168
// 175 and 213 us; E = 32, 48 rows, n = 4096, k = 7168 167 and 242; E = 128, 33 rows, n = 4096, k = 2048 197 and 286.
//
//   warp 0     producer: TMA loads of the token tile and the weight tile per K block
//   warp 1     TMEM allocation; one elected thread issues the MMAs (warp 2 has no role)
//   warp 3     work list: decodes this CTA's tiles one after the other and hands them to the other roles through a
//              queue in shared memory (with every role decoding for itself a tile of two K blocks spent most of its
//              time there)
//   warps 4-19 promotion and output: four TMEM lane quadrants x four column groups; each thread reads the scales of its
//              own token from global memory, four K blocks at a time and four ahead
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "epilogue.cuh"
#include "fp8_blockwise_call.cuh"
#include "mxfp8_quant_math.cuh"
#include "sm100_ptx.cuh"
#include "tensormap.cuh"

namespace es_b200 {
namespace bw {
namespace many {

constexpr int THREADS = 640;
constexpr int EPI_WARP0 = 4, EPI_WARPS = 16;
constexpr int TILE_M = 128;          // token rows per tile
constexpr int TILE_N = 128;          // output columns per tile
constexpr int TILE_K = 128;
constexpr int X_BYTES = TILE_M * TILE_K;
constexpr int STAGE_BYTES = X_BYTES + TILE_N * TILE_K;
constexpr int STAGES = 6;
constexpr int PARTS = 4;             // TMEM partial buffers
constexpr int GROUP_COLS = TILE_N / 4;   // columns of one epilogue warp
constexpr int QUEUE_DEPTH = 4;
constexpr int SCALES_AHEAD = 4;      // K blocks per read of the scales
constexpr int ODD_K_BLOCKS = 10;     // odd numbers of K blocks below this: one K block per hand-over
constexpr uint32_t TMEM_COLS = 512;
// Registers: the kernel is launched with 96 per thread (20 warps); the epilogue warps (32 accumulators, 32 values on their
// way from TMEM, scales of eight K blocks) take over what the other four do not need: 16 x 112 + 4 x 32 = 20 x 96.
constexpr int LAUNCH_REGS = 96, EPI_REGS = 112, ROLE_REGS = 32;
static_assert(EPI_WARPS * EPI_REGS + 4 * ROLE_REGS <= 20 * LAUNCH_REGS, "setmaxnreg only moves the block's registers");

constexpr uint32_t ERR_PRODUCER = 0x1000u, ERR_MMA = 0x2000u, ERR_EPILOGUE = 0x4000u, ERR_WORK_LIST = 0x8000u;

// One tile as the work list hands it out; valid == 0 ends the list.
struct __align__(16) Tile {
  int row0;       // first token row in a / d
  int valid;      // token rows (1 .. 128)
  int col0;       // first output column
  int w_row;      // first weight row in b
};

struct SharedCtl {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t part_full[PARTS];      // one for the partials of a hand-over
  uint64_t part_empty[PARTS];     // one arrival per epilogue warp
  uint64_t q_full[QUEUE_DEPTH];     // 1 arrival: the work-list lane has written the entry
  uint64_t q_empty[QUEUE_DEPTH];    // producer, MMA thread, 16 epilogue warps have read it
  Tile tile[QUEUE_DEPTH];
  uint32_t tmem_base;
  int abort_flag;
  int warp_sums[32];
  int tile_prefix[ES_B200_MAX_EXPERTS + 1];   // tile prefix [0, E], then the per-expert tables (fill_expert_table)
};

constexpr size_t SMEM_BYTES = 1024 + (size_t)STAGES * STAGE_BYTES + sizeof(SharedCtl);
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA per SM");

__device__ uint32_t g_status = 0;

// A consumer's place in the tile queue.
struct QueueReader {
  int qs = 0;
  uint32_t qph = 0;
  __device__ __forceinline__ bool wait(SharedCtl* ctl, volatile int* abort_flag) {
    return ptx::mbar_wait(&ctl->q_full[qs], qph, abort_flag);
  }
  __device__ __forceinline__ const Tile& entry(const SharedCtl* ctl) const { return ctl->tile[qs]; }
  // one arrival per consumer, after its last read of the entry
  __device__ __forceinline__ void release(SharedCtl* ctl) {
    ptx::mbar_arrive(&ctl->q_empty[qs]);
    advance();
  }
  __device__ __forceinline__ void advance() {
    if (++qs == QUEUE_DEPTH) { qs = 0; qph ^= 1u; }
  }
};

__device__ __forceinline__ void give_up(volatile int* abort_flag, uint32_t bit) {
  *abort_flag = 1;
  atomicOr(&g_status, bit);
}

// four consecutive scales: one 16-byte read where every row of them starts on a 16-byte boundary
__device__ __forceinline__ void read_scales(const float* p, int left, bool vec4, float (&v)[SCALES_AHEAD]) {
  if (vec4) {
    const float4 f = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
#pragma unroll
    for (int i = 0; i < SCALES_AHEAD; ++i) v[i] = i < left ? __ldg(p + i) : 0.f;
  }
}

// sixteen columns of a partial, times the scale, onto the accumulators from acc[first] on
__device__ __forceinline__ void promote(const uint32_t (&v)[16], float2 scale, float2 (&acc)[GROUP_COLS / 2], int first) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    acc[first + j] = fma2(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), scale, acc[first + j]);
}

// HAND: K blocks per hand-over from the MMA thread to the promotion: two, but one where a tile has an odd number of K blocks
// below ten, of which the last would take a round trip for itself.  us per call with two and with one: k = 128 (16000 rows,
// 64 experts, n = 4096) 49.1 and 45.8; 384 (21460 Zipf rows, 18, 2816) 61.3 and 57.1; 640 (8000, 64, 2048) 38.8 and 37.1; 896
// 44.4 and 43.3; 1152 52.2 and 51.8; 1664 62.0 both.
template <typename OutT, int HAND>
__global__ void __launch_bounds__(THREADS, 1)
fp8_blockwise_many_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x16,
                               const __grid_constant__ CUtensorMap map_x32, const __grid_constant__ CUtensorMap map_x64,
                               const __grid_constant__ CUtensorMap map_x128, const float* __restrict__ scales_a,
                               const float* __restrict__ scales_b, OutT* __restrict__ d,
                               const int* __restrict__ problem_sizes, const int* __restrict__ expert_offsets,
                               int num_experts, int n, int k, int wide_stores, int scales_vec4) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = ptx::align1024(smem_raw);
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(smem + (size_t)STAGES * STAGE_BYTES);
  const int kt_count = k / TILE_K;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // not the first kernel of its call: the few-rows kernel has waited for the stream's earlier work before it let this
  // one start, so the operands are final; whatever follows may launch at once
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&ctl->full[s], 1);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
    for (int p = 0; p < PARTS / HAND; ++p) {
      ptx::mbar_init(&ctl->part_full[p], 1);
      ptx::mbar_init(&ctl->part_empty[p], EPI_WARPS);
    }
    for (int q = 0; q < QUEUE_DEPTH; ++q) {
      ptx::mbar_init(&ctl->q_full[q], 1);
      ptx::mbar_init(&ctl->q_empty[q], 2 + EPI_WARPS);
    }
    ctl->abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_w);
    ptx::prefetch_tensormap(&map_x16);
    ptx::prefetch_tensormap(&map_x32);
    ptx::prefetch_tensormap(&map_x64);
    ptx::prefetch_tensormap(&map_x128);
  }
  const int col_tiles = n / TILE_N;
  block_exclusive_scan(num_experts, ctl->tile_prefix, ctl->warp_sums, [&](int e) {
    const int m = problem_sizes[e * 3];
    return m > FEW_ROWS ? ((m + TILE_M - 1) / TILE_M) * col_tiles : 0;
  });
  if (ctl->tile_prefix[num_experts] == 0) {      // the host only knows an upper bound of the rows per expert
    pdl_wait_prior_grid();
    return;
  }
  if (warp == 1) {
    ptx::tmem_alloc(&ctl->tmem_base, TMEM_COLS);
    ptx::tmem_relinquish();
  }
  const ExpertTable tab = fill_expert_table(ctl->tile_prefix, num_experts, problem_sizes, expert_offsets, nullptr);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();

  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abort_flag = &ctl->abort_flag;

  if (warp < EPI_WARP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ROLE_REGS));
    if (warp == 3) {
      // ------------------------------------------------------------------ work list: tiles block, block + grid, ...
      // (consecutive tiles, which run at the same time on different SMs, share a weight tile).  A decode — binary search
      // over the experts, a division — takes over a thousand cycles: each lane decodes one of the next 32 tiles.
      const int total = tab.prefix[num_experts];
      int qs = 0;
      uint32_t qph = 0;
      bool ok = true;
      for (int t0 = (int)blockIdx.x; ok; t0 += 32 * (int)gridDim.x) {
        Tile ti = {};
        const int t = t0 + lane * (int)gridDim.x;
        if (t < total) {
          const int e = upper_bound_expert(tab.prefix, num_experts, t);
          const int i = t - tab.prefix[e];
          const int m = tab.m(e);
          const int token_tiles = (m + TILE_M - 1) / TILE_M;
          const int ct = i / token_tiles;
          const int tt = i - ct * token_tiles;
          ti.row0 = tab.row0(e) + tt * TILE_M;
          ti.valid = min(m - tt * TILE_M, TILE_M);
          ti.col0 = ct * TILE_N;
          ti.w_row = e * n + ti.col0;
        }
        __syncwarp();
        const int last = total - t0 <= 0 ? 0 : min(31, (total - t0 - 1) / (int)gridDim.x + 1);   // entries of this batch - 1
        for (int l = 0; l <= last; ++l) {
          if (lane == l) {
            ok = ptx::mbar_wait(&ctl->q_empty[qs], qph ^ 1u, abort_flag);
            if (ok) {
              ctl->tile[qs] = ti;
              ptx::mbar_arrive(&ctl->q_full[qs]);
            }
          }
          ok = __shfl_sync(0xffffffffu, (int)ok, l) != 0;
          if (!ok) break;
          if (++qs == QUEUE_DEPTH) { qs = 0; qph ^= 1u; }
        }
        if (!ok && lane == 0) give_up(abort_flag, ERR_WORK_LIST);
        if (__any_sync(0xffffffffu, t >= total)) break;      // the batch held the end mark
      }
    } else if (warp <= 1 && ptx::elect_one()) {
      if (warp == 0) {
        // ---------------------------------------------------------------- producer
        QueueReader queue;
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        while (ok) {
          if (!queue.wait(ctl, abort_flag)) { ok = false; break; }
          const int valid = queue.entry(ctl).valid, row0 = queue.entry(ctl).row0, w_row = queue.entry(ctl).w_row;
          queue.release(ctl);
          if (valid == 0) break;
          const CUtensorMap* xm = valid <= 16 ? &map_x16 : valid <= 32 ? &map_x32 : valid <= 64 ? &map_x64 : &map_x128;
          const uint32_t box_rows = valid <= 16 ? 16u : valid <= 32 ? 32u : valid <= 64 ? 64u : 128u;
          const uint32_t tx = (box_rows + TILE_N) * TILE_K;
          for (int kt = 0; kt < kt_count; ++kt) {
            if (!ptx::mbar_wait(&ctl->empty[s], ph ^ 1u, abort_flag)) { ok = false; break; }
            uint8_t* stage = smem + (size_t)s * STAGE_BYTES;
            ptx::mbar_arrive_expect_tx(&ctl->full[s], tx);
            ptx::tma_load_2d(stage + X_BYTES, &map_w, &ctl->full[s], kt * TILE_K, w_row);
            ptx::tma_load_2d(stage, xm, &ctl->full[s], kt * TILE_K, row0);
            if (++s == STAGES) { s = 0; ph ^= 1u; }
          }
        }
        if (!ok) give_up(abort_flag, ERR_PRODUCER);
      } else {
        // ---------------------------------------------------------------- MMA issue.  Token rows past the tile's valid
        // ones multiply whatever the stage held before: their lanes of the accumulator are never read.
        const uint32_t idesc = ptx::make_idesc_f8(TILE_M, TILE_N);
        const uint64_t desc0 = ptx::make_desc_k_sw128(ptx::smem_u32(smem));
        QueueReader queue;
        int s = 0, p = 0;                    // stage of the next K block, partials of the next hand-over
        uint32_t ph = 0, p_ph = 0;
        bool ok = true;
        while (ok) {
          if (!queue.wait(ctl, abort_flag)) { ok = false; break; }
          const int valid = queue.entry(ctl).valid;
          queue.release(ctl);
          if (valid == 0) break;
          for (int kt = 0; ok && kt < kt_count; kt += HAND) {
            ok = ptx::mbar_wait(&ctl->part_empty[p], p_ph ^ 1u, abort_flag);
            for (int h = 0; ok && h < HAND && kt + h < kt_count; ++h) {
              ok = ptx::mbar_wait(&ctl->full[s], ph, abort_flag);
              if (!ok) break;
              ptx::tc_fence_after_sync();
              const uint64_t x_desc = desc0 + (uint32_t)(s * (STAGE_BYTES / 16));
              const uint64_t w_desc = x_desc + X_BYTES / 16;
              const uint32_t part = tmem_base + (HAND * p + h) * TILE_N;
#pragma unroll
              for (uint32_t j = 0; j < 4; ++j) ptx::tc_mma_f8(part, x_desc + 2 * j, w_desc + 2 * j, idesc, j != 0 ? 1u : 0u);
              ptx::tc_commit(&ctl->empty[s]);
              if (++s == STAGES) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
            ptx::tc_commit(&ctl->part_full[p]);
            if (++p == PARTS / HAND) { p = 0; p_ph ^= 1u; }
          }
        }
        if (!ok) give_up(abort_flag, ERR_MMA);
      }
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------------------- promotion and output
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPI_REGS));
    constexpr int COLS = GROUP_COLS;
    const int quad = warp & 3;                            // TMEM lane quadrant = 32 token rows
    const int group_col = ((warp - EPI_WARP0) >> 2) * COLS;
    const uint32_t taddr0 = tmem_base + group_col + ((uint32_t)(quad * 32) << 16);
    const bool vec4 = scales_vec4 != 0;
    QueueReader queue;
    int p = 0;
    uint32_t p_ph = 0;
    bool ok = __all_sync(0xffffffffu, queue.wait(ctl, abort_flag));
    // The scales of a tile's first K blocks are requested before the previous tile is stored, the following ones four K
    // blocks ahead.
    int valid = 0, row0 = 0, col0 = 0;
    bool active = false;
    const float *sa = scales_a, *sb = scales_b;
    float sa_next[SCALES_AHEAD], sb_next[SCALES_AHEAD];
#pragma unroll
    for (int i = 0; i < SCALES_AHEAD; ++i) sa_next[i] = sb_next[i] = 0.f;
    auto read_tile = [&] {
      const Tile& ti = queue.entry(ctl);
      valid = ti.valid;
      row0 = ti.row0;
      col0 = ti.col0 + group_col;
      active = quad * 32 < valid;           // warp-uniform: a warp without rows only keeps the barriers moving
      const int row = quad * 32 + lane < valid ? quad * 32 + lane : 0;
      sa = scales_a + (int64_t)(row0 + row) * kt_count;
      sb = scales_b + (int64_t)(ti.w_row / TILE_N) * kt_count;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&ctl->q_empty[queue.qs]);
      queue.advance();
      if (active) {
        read_scales(sa, kt_count, vec4, sa_next);
        read_scales(sb, kt_count, vec4, sb_next);
      }
    };
    if (ok) read_tile();
    while (ok && valid != 0) {
      float2 acc[COLS / 2];
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) acc[j] = make_float2(0.f, 0.f);
      for (int kt0 = 0; ok && kt0 < kt_count; kt0 += SCALES_AHEAD) {
        float s[SCALES_AHEAD];
#pragma unroll
        for (int i = 0; i < SCALES_AHEAD; ++i) s[i] = sa_next[i] * sb_next[i];
        if (active && kt0 + SCALES_AHEAD < kt_count) {
          read_scales(sa + kt0 + SCALES_AHEAD, kt_count - kt0 - SCALES_AHEAD, vec4, sa_next);
          read_scales(sb + kt0 + SCALES_AHEAD, kt_count - kt0 - SCALES_AHEAD, vec4, sb_next);
        }
#pragma unroll
        for (int i = 0; i < SCALES_AHEAD; i += HAND) {
          if (kt0 + i >= kt_count) break;
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->part_full[p], p_ph, abort_flag));
          if (!ok) break;
          if (active) {
            // Sixteen columns at a time, so that the reads of the next ones are on their way during the multiplications.
            ptx::tc_fence_after_sync();
            const uint32_t taddr = taddr0 + p * HAND * TILE_N;
            const bool two = HAND == 2 && kt0 + i + 1 < kt_count;
            const float2 s0 = make_float2(s[i], s[i]), s1 = make_float2(s[i + HAND - 1], s[i + HAND - 1]);
            uint32_t va[16], vb[16];
            ptx::tc_ld_32x32b_x16(taddr, va);
            ptx::tc_ld_32x32b_x16(taddr + 16, vb);
            ptx::tc_wait_ld();
            promote(va, s0, acc, 0);
            if (two) ptx::tc_ld_32x32b_x16(taddr + TILE_N, va);
            if (HAND == 2) promote(vb, s0, acc, 8);
            if (two) {
              ptx::tc_wait_ld();
              ptx::tc_ld_32x32b_x16(taddr + TILE_N + 16, vb);
              promote(va, s1, acc, 0);
              ptx::tc_wait_ld();
            }
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&ctl->part_empty[p]);   // the tensor core may overwrite these partials
            if (two || HAND == 1) promote(vb, s1, acc, 8);
          } else if (lane == 0) {
            ptx::mbar_arrive(&ctl->part_empty[p]);
          }
          if (++p == PARTS / HAND) { p = 0; p_ph ^= 1u; }
        }
      }
      if (!ok) break;
      const bool store = active && quad * 32 + lane < valid;
      OutT* out = d + (int64_t)(row0 + quad * 32 + lane) * n + col0;
      ok = __all_sync(0xffffffffu, queue.wait(ctl, abort_flag));
      if (ok) read_tile();
      // this thread's columns of its output row, 32 bytes at a time
      if (store) {
#pragma unroll
        for (int j = 0; j < COLS / 16; ++j) {
          uint32_t w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) w[i] = pack_pair_from_f32<OutT>(acc[j * 8 + i].x, acc[j * 8 + i].y);
          store_32B(out + j * 16, w, wide_stores != 0);
        }
      }
    }
    if (!ok && lane == 0) give_up(abort_flag, ERR_EPILOGUE);
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::settle_if_aborted(abort_flag);
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, TMEM_COLS);
  }
  pdl_wait_prior_grid();   // do not complete before the few-rows kernel of this call has
}

template <typename OutT, int HAND>
int launch_as(const CallArgs& c) {
  DeviceInfo info;
  int rc = get_device_info(&info);
  if (rc != ES_B200_OK) return rc;
  CUtensorMap map_w, map_x[4];
  rc = make_tensormap_u8_sw128(&map_w, c.b, (uint64_t)c.num_experts * c.n, (uint64_t)c.k, TILE_N);
  if (rc != ES_B200_OK) return rc;
  const uint32_t boxes[4] = {16, 32, 64, 128};
  for (int i = 0; i < 4; ++i) {
    rc = make_tensormap_u8_sw128(&map_x[i], c.a, (uint64_t)c.num_rows, (uint64_t)c.k, boxes[i]);
    if (rc != ES_B200_OK) return rc;
  }
  auto kernel = fp8_blockwise_many_rows_kernel<OutT, HAND>;
  static bool configured[64] = {false};
  int dev = 0;
  ES_CUDA_TRY(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    // the register hand-over inside the kernel would wait for ever in a block launched with fewer registers
    cudaFuncAttributes attrs;
    ES_CUDA_TRY(cudaFuncGetAttributes(&attrs, kernel));
    if (attrs.numRegs < LAUNCH_REGS)
      return fail(ES_B200_ERR_CUDA, "the blockwise kernel was built with %d registers per thread, %d expected",
                  attrs.numRegs, LAUNCH_REGS);
    ES_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
    configured[dev & 63] = true;
  }
  // upper bound of the tiles that the host can know: full token tiles plus one partial tile per expert, of which at most
  // num_rows / (FEW_ROWS + 1) have work here
  const int64_t by_rows = c.num_rows / (FEW_ROWS + 1);
  const int64_t experts = c.num_experts < by_rows ? c.num_experts : by_rows;
  const int64_t max_tiles = (c.num_rows / TILE_M + experts) * (c.n / TILE_N);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(max_tiles < info.sm_count ? max_tiles : info.sm_count));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int kt_count = c.k / TILE_K;
  const bool vec4 = kt_count % SCALES_AHEAD == 0 && aligned16(c.sa) && aligned16(c.sb);
  ES_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, map_w, map_x[0], map_x[1], map_x[2], map_x[3], c.sa, c.sb,
                                 static_cast<OutT*>(c.d), c.ps, c.eo, c.num_experts, c.n, c.k,
                                 (reinterpret_cast<uintptr_t>(c.d) & 31u) == 0 ? 1 : 0, vec4 ? 1 : 0));
  return ES_B200_OK;
}

template <typename OutT>
int launch(const CallArgs& c) {
  const int kt_count = c.k / TILE_K;
  return (kt_count & 1) != 0 && kt_count < ODD_K_BLOCKS ? launch_as<OutT, 1>(c) : launch_as<OutT, 2>(c);
}

}  // namespace many

int launch_many_rows_bf16(const CallArgs& c) { return many::launch<__nv_bfloat16>(c); }
int launch_many_rows_fp16(const CallArgs& c) { return many::launch<__half>(c); }

int read_and_clear_status_many_rows(uint32_t* out) {
  uint32_t v = 0;
  ES_CUDA_TRY(cudaMemcpyFromSymbol(&v, many::g_status, sizeof(v)));
  if (v != 0) {
    uint32_t zero = 0;
    ES_CUDA_TRY(cudaMemcpyToSymbol(many::g_status, &zero, sizeof(zero)));
  }
  *out = v;
  return ES_B200_OK;
}

}  // namespace bw
}  // namespace es_b200
