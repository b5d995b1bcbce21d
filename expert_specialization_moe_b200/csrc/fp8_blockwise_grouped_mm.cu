// FP8-blockwise grouped GEMM for sm_100a: e4m3 x e4m3 with fp32 scales (one per 1x128 of a, one per 128x128 of b).
//
// Per expert e:  d[off_e + i, n] = sum_kb sa[off_e + i, kb] * sb[e, n/128, kb] * sum_{k in kb} a[off_e + i, k] * b[e, n, k]
//
// The reference runs this op on Hopper only (wgmma templates).  Here every 128-wide K block is one unscaled
// tcgen05.mma.kind::f8f6f4 group (4 MMAs of K=32) into a TMEM partial buffer; the epilogue warps pull each partial out
// of TMEM (tcgen05.ld), multiply by the block's scale product and accumulate in fp32 registers while the tensor core
// works on the following K blocks (two-stage promotion, as the reference's Hopper kernel does in registers).  Work list
// from a per-CTA prefix scan, persistent grids of one CTA per SM; two launches chained with programmatic dependent
// launch, each taking the experts of its row counts:
//   few_rows  (<= 32 rows) 128 WEIGHT rows on the MMA M axis, the expert's tokens on its N axis.  Bound by HBM on the
//             weights: what counts is bytes in flight (10 stages of 20 KB) and little shared-memory traffic besides;
//   many_rows (>= 33 rows) 128 TOKEN rows on the M axis, 128 weight rows on the N axis.  A TMEM lane is then one
//             token, so the scale of a K block is ONE register per thread: the promotion is a packed FMA with a scalar,
//             without the broadcast shared-memory read per four FMAs that the other mapping needs next to the MMAs'
//             operand reads, and a thread ends up with consecutive columns of one output row, stored as 32-byte pieces
//             without a transposition.
//
// This file: the few-rows kernel and the entry point.
//   warp 0     producer: TMA loads of the weight tile and the token tile per K block
//   warps 1, 2 MMA issue, one thread each: warp 1 (which also owns the TMEM allocation) takes the even K blocks, warp 2
//              the odd ones (consecutive K blocks go to different partial buffers); with short K warp 1 alone
//   warps 3, 4 scale loaders, alternating chunks: sa[token, kb] * sb[tile, kb] for 8 K blocks at a time, transposed to
//              [kb][token] in a ring of chunks, so that the epilogue reads one broadcast float4 per 4 tokens and never
//              waits on global memory, whatever K is
//   warps 5-12 promotion (partial * scale -> fp32 registers) and output through a per-warp shared-memory transpose:
//              two groups of four warps (the four TMEM lane quadrants) take alternate tiles, which hides the per-tile
//              latencies (work-list decode, output) that dominate when K is only 2-4 blocks
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "epilogue.cuh"
#include "fp8_blockwise_call.cuh"
#include "sm100_ptx.cuh"
#include "tensormap.cuh"

namespace es_b200 {
namespace bw {

constexpr int TILE_N = 128;          // weight rows per tile
constexpr int TILE_K = 128;
constexpr int TOK = FEW_ROWS;        // token rows per tile = columns of one TMEM partial
constexpr int W_BYTES = TILE_N * TILE_K;
constexpr int STAGE_BYTES = W_BYTES + TOK * TILE_K;
constexpr int STAGES = 10;
constexpr int NPART = 4;             // TMEM partial buffers
constexpr uint32_t TMEM_COLS = NPART * TOK;
constexpr int SHORT_K_BLOCKS = 4;    // fewer K blocks than this: short K
constexpr int CH_KT = 8;             // K blocks per scale chunk
constexpr int NCH = 4;               // scale chunks in the ring
constexpr int CHUNK_FLOATS = CH_KT * TOK;
constexpr int LOADER_WARP0 = 3;      // two scale loaders
constexpr int EPI_WARP0 = 5;
constexpr int GROUP_WARPS = 4;       // epilogue group: the four TMEM lane quadrants; two groups take alternate tiles
constexpr int EPI_WARPS = 2 * GROUP_WARPS;
constexpr int THREADS = 32 * (EPI_WARP0 + EPI_WARPS);
constexpr int EPI_TOK = 16;                          // tokens per pass through an epilogue warp's transposition tile
constexpr int EPI_TILE_BYTES = EPI_TOK * 32 * 2;     // 1 KB

constexpr uint32_t ERR_PRODUCER = 0x1000u, ERR_MMA = 0x2000u, ERR_EPILOGUE = 0x4000u, ERR_SCALES = 0x8000u;

struct SharedCtl {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t part_full[NPART];
  uint64_t part_empty[NPART];     // one arrival per warp of the epilogue group that owns the tile
  uint64_t chunk_full[NCH];       // 1 arrival: the chunk's scale loader
  uint64_t chunk_empty[NCH];      // one arrival per warp of the epilogue group that owns the tile
  uint64_t turn[2];               // turn[x]: epilogue group x may enter the K loop of its next tile
  uint32_t tmem_base;
  int abort_flag;
  int warp_sums[32];
  int tile_prefix[ES_B200_MAX_EXPERTS + 1];   // item prefix [0, E], then the per-expert tables (fill_expert_table)
};

constexpr size_t SMEM_BYTES = 1024 + (size_t)STAGES * STAGE_BYTES + (size_t)NCH * CHUNK_FLOATS * 4 +
                              (size_t)EPI_WARPS * EPI_TILE_BYTES + sizeof(SharedCtl);
static_assert((NCH & (NCH - 1)) == 0 && (NPART & (NPART - 1)) == 0, "ring slots are taken modulo a power of two");
// A waiter may be at most one phase ahead of its mbarrier.  Each ring barrier therefore has ONE waiting role per
// revolution: K blocks (and chunks) alternate between two lanes (warps), so ring sizes must be even.
static_assert(STAGES % 2 == 0 && NPART % 2 == 0 && NCH % 2 == 0, "alternating owners need even rings");
static_assert(STAGE_BYTES % 1024 == 0, "stages must keep the 1024-byte alignment of the swizzled tiles");
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA per SM");

__device__ uint32_t g_status = 0;

struct TileInfo {
  int e, nt, valid, n_mma, row0;
};

// A work item is `group` consecutive weight tiles of one expert; CTA `block` of `blocks` takes the items block, block +
// blocks, ... and every role walks their tiles in the same order.  The item is decoded once (binary search over the item
// prefix) and the tiles inside it only advance `nt`: with two K blocks per tile (k = 256) a decode per tile costs every
// role more time than its work on the tile (the producer lane and both MMA lanes ~2200 cycles, almost none of it waiting).
struct TileWalk {
  TileInfo ti;
  int item, left, blocks;
  __device__ __forceinline__ TileWalk(int block, int blocks_) : item(block - blocks_), left(0), blocks(blocks_) {}
  // advances to this CTA's next tile; false when there is none
  __device__ __forceinline__ bool next(const ExpertTable& tab, int num_experts, int total_items, int n_tiles, int group) {
    if (left > 0) {
      --left;
      ++ti.nt;
      return true;
    }
    item += blocks;
    if (item >= total_items) return false;
    ti.e = upper_bound_expert(tab.prefix, num_experts, item);
    ti.nt = (item - tab.prefix[ti.e]) * group;
    ti.valid = tab.m(ti.e);
    ti.n_mma = (ti.valid + 15) & ~15;
    ti.row0 = tab.row0(ti.e);
    const int rest = n_tiles - ti.nt;
    left = (rest < group ? rest : group) - 1;
    return true;
  }
};

// One CTA per SM; serves the experts with 1 .. FEW_ROWS rows.  First kernel of its call.
// SHORT_K (fewer than four K blocks): ONE thread issues all MMAs, elected (a thread found by lane == 0 needs 550 cycles for
// the four MMAs, waits and commits of a K block, an elected one 350, and K blocks then need no second thread).  Per call,
// two threads and one: 4096 rows on 256 experts, n = 7168, k = 256 91.8 and 87.3 us; 1500 Zipf rows on 128, n = 4096, k = 384
// 45.2 and 43.3; but 2000 rows on 256, n = 4096, k = 512 92.2 and 94.3; E = 256, n = 512, k = 7168 149.8 and 153.3: bound by
// HBM, which a quicker turn-round of the stages does not suit.
template <typename OutT, bool SHORT_K>
__global__ void __launch_bounds__(THREADS, 1)
fp8_blockwise_grouped_mm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x16,
                                const __grid_constant__ CUtensorMap map_x32, const float* scales_a,
                                const float* scales_b, OutT* __restrict__ d,
                                const int* problem_sizes, const int* expert_offsets,
                                int num_experts, int n, int k, int group) {
  const int block = (int)blockIdx.x, blocks = (int)gridDim.x;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = ptx::align1024(smem_raw);
  float* chunks = reinterpret_cast<float*>(smem + (size_t)STAGES * STAGE_BYTES);        // [NCH][CH_KT][TOK]
  uint8_t* epi_stage = reinterpret_cast<uint8_t*>(chunks + NCH * CHUNK_FLOATS);        // 1 KB per epilogue warp
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(epi_stage + (size_t)EPI_WARPS * EPI_TILE_BYTES);
  const int kt_count = k / TILE_K;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&ctl->full[s], 1);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
    for (int p = 0; p < NPART; ++p) {
      ptx::mbar_init(&ctl->part_full[p], 1);
      ptx::mbar_init(&ctl->part_empty[p], GROUP_WARPS);
    }
    for (int c = 0; c < NCH; ++c) {
      ptx::mbar_init(&ctl->chunk_full[c], 1);
      ptx::mbar_init(&ctl->chunk_empty[c], GROUP_WARPS);
    }
    ptx::mbar_init(&ctl->turn[0], GROUP_WARPS);
    ptx::mbar_init(&ctl->turn[1], GROUP_WARPS);
    ctl->abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&map_w);
    ptx::prefetch_tensormap(&map_x16);
    ptx::prefetch_tensormap(&map_x32);
  }
  if (warp == 1) {
    ptx::tmem_alloc(&ctl->tmem_base, TMEM_COLS);
    ptx::tmem_relinquish();
  }
  // This kernel waits for the stream's earlier work and then lets the many-rows kernel of the call start; that one writes
  // other rows of d and only waits for this one before it exits (stream order).
  pdl_wait_prior_grid();
  const int n_tiles = n / TILE_N;
  block_exclusive_scan(num_experts, ctl->tile_prefix, ctl->warp_sums, [&](int e) {
    const int m = problem_sizes[e * 3];
    return (m > 0 && m <= FEW_ROWS) ? (n_tiles + group - 1) / group : 0;
  });
  // a launch without work (the host only knows an upper bound of the rows per expert) ends here
  if (ctl->tile_prefix[num_experts] == 0) {
    pdl_launch_dependents();
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) ptx::tmem_dealloc(ctl->tmem_base, TMEM_COLS);
    return;
  }
  const ExpertTable tab = fill_expert_table(ctl->tile_prefix, num_experts, problem_sizes, expert_offsets, nullptr);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  pdl_launch_dependents();

  const uint32_t tmem_base = ctl->tmem_base;
  const int total_items = ctl->tile_prefix[num_experts];
  volatile int* abort_flag = &ctl->abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      TileWalk walk(block, blocks);
      while (ok && walk.next(tab, num_experts, total_items, n_tiles, group)) {
        const TileInfo& ti = walk.ti;
        const CUtensorMap* xm = ti.n_mma <= 16 ? &map_x16 : &map_x32;
        const uint32_t box_rows = ti.n_mma <= 16 ? 16u : 32u;
        const uint32_t tx = W_BYTES + box_rows * TILE_K;
        const int w_row = ti.e * n + ti.nt * TILE_N;
        for (int kt = 0; kt < kt_count; ++kt) {
          if (!ptx::mbar_wait(&ctl->empty[s], ph ^ 1u, abort_flag)) {
            ok = false;
            *abort_flag = 1;
            atomicOr(&g_status, ERR_PRODUCER);
            break;
          }
          uint8_t* stage = smem + (size_t)s * STAGE_BYTES;
          ptx::mbar_arrive_expect_tx(&ctl->full[s], tx);
          ptx::tma_load_2d(stage, &map_w, &ctl->full[s], kt * TILE_K, w_row);
          ptx::tma_load_2d(stage + W_BYTES, xm, &ctl->full[s], kt * TILE_K, ti.row0);
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 1 || warp == 2) {
    // ------------------------------------------------------------------ MMA issue; g counts K blocks over all tiles of this
    // CTA (stage = g mod STAGES, partial = g mod 4).  With long K the K blocks alternate between the two threads.
    auto issue = [&](int mine) {
      int g = 0;
      bool ok = true;
      TileWalk walk(block, blocks);
      while (ok && walk.next(tab, num_experts, total_items, n_tiles, group)) {
        const TileInfo& ti = walk.ti;
        const uint32_t idesc = ptx::make_idesc_f8(TILE_N, ti.n_mma);
        for (int kt = 0; kt < kt_count; ++kt, ++g) {
          if (!SHORT_K && (g & 1) != mine) continue;
          const int s = g % STAGES;
          const uint32_t ph = (uint32_t)(g / STAGES) & 1u;
          const int p = g & (NPART - 1);
          const uint32_t p_ph = (uint32_t)(g / NPART) & 1u;
          if (!ptx::mbar_wait(&ctl->part_empty[p], p_ph ^ 1u, abort_flag)) { ok = false; break; }
          if (!ptx::mbar_wait(&ctl->full[s], ph, abort_flag)) { ok = false; break; }
          ptx::tc_fence_after_sync();
          const uint32_t stage = ptx::smem_u32(smem + (size_t)s * STAGE_BYTES);
          const uint64_t a_desc = ptx::make_desc_k_sw128(stage);
          const uint64_t b_desc = ptx::make_desc_k_sw128(stage + W_BYTES);
          const uint32_t d_tmem = tmem_base + p * TOK;
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j)
            ptx::tc_mma_f8(d_tmem, a_desc + 2 * j, b_desc + 2 * j, idesc, j != 0 ? 1u : 0u);
          ptx::tc_commit(&ctl->empty[s]);
          ptx::tc_commit(&ctl->part_full[p]);
        }
        if (!ok) {
          *abort_flag = 1;
          atomicOr(&g_status, ERR_MMA);
        }
      }
    };
    if constexpr (SHORT_K) {
      if (warp == 1 && ptx::elect_one()) issue(0);
    } else {
      if (lane == 0) issue(warp - 1);
    }
  } else if (warp < EPI_WARP0) {
    // ------------------------------------------------------------------ scale loaders: chunks alternate between the
    // two warps; c counts chunks over all tiles of this CTA (ring slot = c mod NCH)
    const int mine = warp - LOADER_WARP0;
    int c = 0;
    bool ok = true;
    TileWalk walk(block, blocks);
    while (ok && walk.next(tab, num_experts, total_items, n_tiles, group)) {
      const int chunks_in_tile = (kt_count + CH_KT - 1) / CH_KT;
      // this warp's chunks of the tile: c, c+1, .. with (c & 1) == mine
      if (chunks_in_tile == 1 && (c & 1) != mine) { ++c; continue; }   // common for small K
      const TileInfo& ti = walk.ti;
      const float* sb_row = scales_b + ((int64_t)ti.e * n_tiles + ti.nt) * kt_count;
      for (int kt0 = 0; kt0 < kt_count; kt0 += CH_KT, ++c) {
        if ((c & 1) != mine) continue;
        const int cs = c & (NCH - 1);
        const uint32_t c_ph = (uint32_t)(c / NCH) & 1u;
        // the loads do not depend on the ring slot: issue them before waiting for it
        const int nk = kt_count - kt0 < CH_KT ? kt_count - kt0 : CH_KT;
        float sb[CH_KT];
#pragma unroll
        for (int i = 0; i < CH_KT; ++i) sb[i] = i < nk ? sb_row[kt0 + i] : 0.f;
        float sa[CH_KT];                           // of token `lane`
        const float* sa_row = scales_a + (int64_t)(ti.row0 + lane) * kt_count + kt0;
#pragma unroll
        for (int i = 0; i < CH_KT; ++i) sa[i] = (lane < ti.valid && i < nk) ? sa_row[i] : 0.f;
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctl->chunk_empty[cs], c_ph ^ 1u, abort_flag))) {
          ok = false;
          if (lane == 0) {
            *abort_flag = 1;
            atomicOr(&g_status, ERR_SCALES);
          }
          break;
        }
        float* chunk = chunks + cs * CHUNK_FLOATS;
#pragma unroll
        for (int i = 0; i < CH_KT; ++i) chunk[i * TOK + lane] = sa[i] * sb[i];
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&ctl->chunk_full[cs]);
      }
    }
  } else {
    // ------------------------------------------------------------------ promotion and output (warps 5..)
    // Consecutive tiles alternate between the epilogue groups: while one group converts and stores its tile (and
    // decodes the next), the other is already accumulating the following tile's partials.  The K loops themselves
    // are strictly serial (turn barriers): a group that waited on part_full / chunk_full for a tile further ahead
    // would be more than one phase ahead of those barriers, and a parity wait cannot tell phases n and n+2 apart.
    const int q = warp & 3;                           // TMEM lane quadrant of this warp
    const int egroup = (warp - EPI_WARP0) / GROUP_WARPS;
    OutT* stage_warp = reinterpret_cast<OutT*>(epi_stage) + (warp - EPI_WARP0) * (EPI_TOK * 32);
    const int part = lane & 3;
    int g = 0;                                        // K blocks over all tiles of this CTA
    int c = 0;                                        // scale chunks over all tiles of this CTA
    bool alive = true;
    uint32_t turn_ph = 0;
    int tile_index = 0;
    TileWalk walk(block, blocks);
    while (alive && walk.next(tab, num_experts, total_items, n_tiles, group)) {
      const int my_index = tile_index++;
      if ((my_index & 1) != egroup) {   // the other group's tile
        g += kt_count;
        c += (kt_count + CH_KT - 1) / CH_KT;
        continue;
      }
      const TileInfo& ti = walk.ti;
      float acc[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = 0.f;
      if (my_index > 0) {                              // the other group has left the K loop of the previous tile
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctl->turn[egroup], turn_ph, abort_flag))) {
          if (lane == 0) {
            *abort_flag = 1;
            atomicOr(&g_status, ERR_EPILOGUE);
          }
          break;
        }
        turn_ph ^= 1u;
      }

      for (int kt = 0; kt < kt_count; ++kt, ++g) {
        const int ki = kt & (CH_KT - 1);
        const int cs = c & (NCH - 1);
        const int p = g & (NPART - 1);
        bool got = true;
        if (ki == 0) got = ptx::mbar_wait(&ctl->chunk_full[cs], (uint32_t)(c / NCH) & 1u, abort_flag);
        got = got && ptx::mbar_wait(&ctl->part_full[p], (uint32_t)(g / NPART) & 1u, abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) {
            *abort_flag = 1;
            atomicOr(&g_status, ERR_EPILOGUE);
          }
          alive = false;
          break;
        }
        uint32_t v[32];
        ptx::tc_fence_after_sync();
        ptx::tc_ld_32x32b_x32(tmem_base + p * TOK + ((uint32_t)(q * 32) << 16), v);
        ptx::tc_wait_ld();
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&ctl->part_empty[p]);      // the tensor core may overwrite this partial
        const float4* srow = reinterpret_cast<const float4*>(chunks + cs * CHUNK_FLOATS + ki * TOK);
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          const float4 sc = srow[j4];                  // same address in every lane: broadcast
          acc[j4 * 4 + 0] = fmaf(__uint_as_float(v[j4 * 4 + 0]), sc.x, acc[j4 * 4 + 0]);
          acc[j4 * 4 + 1] = fmaf(__uint_as_float(v[j4 * 4 + 1]), sc.y, acc[j4 * 4 + 1]);
          acc[j4 * 4 + 2] = fmaf(__uint_as_float(v[j4 * 4 + 2]), sc.z, acc[j4 * 4 + 2]);
          acc[j4 * 4 + 3] = fmaf(__uint_as_float(v[j4 * 4 + 3]), sc.w, acc[j4 * 4 + 3]);
        }
        if (ki == CH_KT - 1 || kt == kt_count - 1) {          // done with this scale chunk
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&ctl->chunk_empty[cs]);
          ++c;
        }
      }
      if (!alive) break;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&ctl->turn[egroup ^ 1]);
      // output: this warp's 32 n of up to 32 tokens, 16 tokens at a time through its 1 KB tile, 128-bit stores (4 lanes per
      // 64-byte row piece)
      OutT* dst = d + (int64_t)ti.row0 * n + (ti.nt * TILE_N + q * 32);
#pragma unroll
      for (int h = 0; h < TOK / EPI_TOK; ++h) {
#pragma unroll
        for (int j = 0; j < EPI_TOK; ++j) stage_warp[j * 32 + lane] = out_from_f32<OutT>(acc[h * EPI_TOK + j]);
        __syncwarp();
#pragma unroll
        for (int it = 0; it < EPI_TOK / 8; ++it) {
          const int tok = it * 8 + (lane >> 2);
          const uint4 val = *reinterpret_cast<const uint4*>(stage_warp + tok * 32 + part * 8);
          const int row = h * EPI_TOK + tok;
          if (row < ti.valid) *reinterpret_cast<uint4*>(dst + (int64_t)row * n + part * 8) = val;
        }
        __syncwarp();
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::settle_if_aborted(abort_flag);
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// weight tiles per work item: the per-item work of every role (decode) is spread over ~8 K blocks
static int tiles_per_item(int k) {
  const int kt_count = k / TILE_K;
  const int group = (8 + kt_count - 1) / kt_count;
  return group < 1 ? 1 : group;
}

template <typename OutT, bool SHORT_K>
int launch_few_rows_as(const CallArgs& c) {
  DeviceInfo info;
  int rc = get_device_info(&info);
  if (rc != ES_B200_OK) return rc;
  CUtensorMap map_w, map_x16, map_x32;
  rc = make_tensormap_u8_sw128(&map_w, c.b, (uint64_t)c.num_experts * c.n, (uint64_t)c.k, TILE_N);
  if (rc == ES_B200_OK) rc = make_tensormap_u8_sw128(&map_x16, c.a, (uint64_t)c.num_rows, (uint64_t)c.k, 16);
  if (rc == ES_B200_OK) rc = make_tensormap_u8_sw128(&map_x32, c.a, (uint64_t)c.num_rows, (uint64_t)c.k, 32);
  if (rc != ES_B200_OK) return rc;
  auto kernel = fp8_blockwise_grouped_mm_kernel<OutT, SHORT_K>;
  static bool configured[64] = {false};
  int dev = 0;
  ES_CUDA_TRY(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    ES_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES));
    configured[dev & 63] = true;
  }
  const int group = tiles_per_item(c.k);
  // one CTA per SM, fewer when the host-known upper bound of the item count is smaller
  const int64_t experts = c.num_experts < c.num_rows ? c.num_experts : c.num_rows;
  const int64_t max_items = experts * ((c.n / TILE_N + group - 1) / group);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(max_items < info.sm_count ? max_items : info.sm_count));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ES_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, map_w, map_x16, map_x32, c.sa, c.sb, static_cast<OutT*>(c.d), c.ps, c.eo,
                                 c.num_experts, c.n, c.k, group));
  return ES_B200_OK;
}

template <typename OutT>
int launch_few_rows(const CallArgs& c) {
  return c.k / TILE_K < SHORT_K_BLOCKS ? launch_few_rows_as<OutT, true>(c) : launch_few_rows_as<OutT, false>(c);
}

int read_and_clear_status(uint32_t* out) {
  uint32_t v = 0, many = 0;
  ES_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_status, sizeof(v)));
  if (v != 0) {
    uint32_t zero = 0;
    ES_CUDA_TRY(cudaMemcpyToSymbol(g_status, &zero, sizeof(zero)));
  }
  const int rc = read_and_clear_status_many_rows(&many);
  *out = v | many;
  return rc;
}

}  // namespace bw
}  // namespace es_b200

extern "C" int es_b200_fp8_blockwise_grouped_mm(const void* a, const void* b, const float* scales_a,
                                                const float* scales_b, void* d, int out_dtype,
                                                const int32_t* problem_sizes, const int32_t* expert_offsets,
                                                int num_experts, int64_t num_rows, int n, int k, void* scratch,
                                                size_t scratch_bytes, void* stream) {
  es_b200::NvtxRange nvtx_range("es_b200_fp8_blockwise_grouped_mm");
  using namespace es_b200;
  (void)scratch; (void)scratch_bytes;
  ES_REQUIRE(out_dtype == ES_B200_BF16 || out_dtype == ES_B200_FP16, "output must be bfloat16 or half");
  ES_REQUIRE(k > 0 && k % 128 == 0, "k should align 128");
  ES_REQUIRE(n > 0 && n % 128 == 0, "n should align 128");
  ES_REQUIRE(num_experts >= 0 && num_experts <= ES_B200_MAX_EXPERTS, "Number of experts cannot exceed %d",
             ES_B200_MAX_EXPERTS);
  ES_REQUIRE(num_rows >= 0 && num_rows < (int64_t)1 << 31, "num_rows out of range");
  ES_REQUIRE((int64_t)num_experts * n < (int64_t)1 << 31, "num_experts * n out of range");
  if (num_experts == 0 || num_rows == 0) return ES_B200_OK;
  ES_REQUIRE(a && b && scales_a && scales_b && d && problem_sizes && expert_offsets, "null pointer argument");
  ES_REQUIRE(aligned16(a) && aligned16(b) && aligned16(d), "a, b and d must be 16-byte aligned");
  ES_REQUIRE((reinterpret_cast<uintptr_t>(scales_a) & 3u) == 0 && (reinterpret_cast<uintptr_t>(scales_b) & 3u) == 0,
             "scales must be 4-byte aligned");
  // The few-rows kernel first, then the many-rows kernel; every CTA filters the experts in its own scan.  A bucket that
  // even the host-known upper bound of rows per expert cannot reach gets no launch.
  const bw::CallArgs c = {a, b, scales_a, scales_b, d, problem_sizes, expert_offsets, num_experts, num_rows, n, k,
                          static_cast<cudaStream_t>(stream)};
  const bool bf16 = out_dtype == ES_B200_BF16;
  const int rc = bf16 ? bw::launch_few_rows<__nv_bfloat16>(c) : bw::launch_few_rows<__half>(c);
  if (rc != ES_B200_OK || num_rows <= bw::FEW_ROWS) return rc;
  return bf16 ? bw::launch_many_rows_bf16(c) : bw::launch_many_rows_fp16(c);
}
