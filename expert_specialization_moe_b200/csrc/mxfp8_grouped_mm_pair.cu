// The kernel of the MXFP8 block-scaled grouped GEMM for sm_100a: CTA pairs (tcgen05.mma.cta_group::2), persistent, one
// launch per call for experts of any row count.
//
// Mapping: weights on the MMA M axis, the expert's token rows on the runtime-sized N axis (a multiple of 16: 3 rows cost an
// N = 16 MMA, no padding of the ragged dimension to 128).  Two CTAs of a cluster share every work item: 256 weight rows —
// each CTA holds 128 — times up to 384 token rows, half of them in each CTA's shared memory; the pair's tensor cores exchange
// the halves (no multicast load anywhere).  More than 192 token rows are two sub-tiles with an accumulator each, so that
// every 16 KB weight tile that a CTA pulls through L2 feeds both; up to 192 rows are one sub-tile and the two accumulators
// take turns.  An expert's rows are divided into token tiles of whole 128-row scale atoms, as evenly as they go.
//
// What bounds it.  Experts of few rows stream their weights from HBM once: 1.69 GB in 239 us = 7.1 TB/s (256 experts, 512
// rows, n = 7168, k = 2048).  Experts of many rows: the tensor pipe (a K step of 384 rows is 768 cycles of it, 782 measured),
// then the power cap.  In between (about 256 rows): the K steps of token rows in flight (128 experts x 256 rows, n = 1536,
// k = 2048: 158 us with 2 K steps, 124 with 3, 117 with 4).
//
// What it took, measured cycle by cycle on its predecessor (three launches per call, 72 to 105 us more for the layer's two
// GEMMs):
//   * tcgen05 and TMA instructions are issued by a thread that elect.sync picked.  Guarded by lane == 0 the same code
//     needs 137 cycles per MMA and 550 per K step; elected, MMAs go out at the pipe's rate (40 cycles at N = 16);
//   * one barrier wait (130 cycles) and one commit (90) per K step: what a K step cannot have is several of them in a row;
//   * arrivals at the partner CTA that publish no memory are relaxed: a releasing one first waits for the epilogue's
//     stores, 2000 to 3000 cycles before every hand-back of an accumulator;
//   * work items are decoded once, by a warp that does nothing else, and queued four deep (every role decoded for
//     itself: 2000 cycles per item);
//   * the output leaves as 16-byte stores: matrix fragments from TMEM (16x256b), transposed by stmatrix.
//
// GATED (es_b200_mxfp8_grouped_mm_silu_mul_quant): silu(gate) * up and the requantisation in the epilogue.  A work item is 256
// gate rows, the 256 up rows of the same outputs, and up to 192 token rows; a K step has two weight slots and one token slot,
// gate goes to the first accumulator, up to the second, so that a thread finds both of an output in the same lane and column,
// a warp its 32 outputs of a scale block.  The gate_up product is neither rounded to 16 bits nor written: 128 x 1024 rows,
// inter = 768, k = 2048: 336 us (each kernel timed by a profiler) where the GEMM took 281 and the SiLU kernel 126.
//
//   warp 0      producer of weights and scales (both CTAs): per K step one thread loads its 128 weight rows, their scale atom
//               and the item's token scale atoms; all bytes are credited to the leader CTA's barrier
//   warp 1      TMEM allocation; in the leader CTA one thread issues the K step's scale copies (tcgen05.cp) and MMAs
//   warp 2      scheduler (leader): takes item indices from the work counter and queues the items in both CTAs
//   warp 3      producer of token rows (both CTAs): this CTA's half of each sub-tile
//   warps 4-15  epilogue (both CTAs)
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "epilogue.cuh"
#include "grouped_mm_call.cuh"
#include "mxfp8_quant_math.cuh"
#include "sm100_ptx.cuh"
#include "tensormap.cuh"
#include "work_items.cuh"

namespace es_b200 {
namespace mm {

constexpr int THREADS = 512;
constexpr int TILE_N = 128;      // weight rows per CTA (the pair covers 256)
constexpr int TILE_K = 128;
constexpr int SUB_TILE = 192;    // token rows per accumulator (MMA N, runtime multiple of 16)
constexpr int ITEM_ATOMS = 3;    // 128-row scale atoms per work item: up to 384 token rows
constexpr int W_BYTES = TILE_N * TILE_K;               // 16384
constexpr int SF_BYTES = 512;
constexpr int SFX_BYTES = ITEM_ATOMS * SF_BYTES;
constexpr int W_SLOT = W_BYTES + SF_BYTES + SFX_BYTES; // 18432: W | SFW | SFX
constexpr int X_SLOT = (SUB_TILE / 2) * TILE_K;        // 12288: this CTA's half of one token sub-tile
static_assert(W_SLOT % 1024 == 0 && X_SLOT % 1024 == 0, "128-byte swizzle atoms are 1024 bytes");
// The two rings share what shared memory there is: W weight slots (one per K step), X token slots (one per sub-tile of a K
// step).  Few rows per expert: seven K steps in flight.  Many: eight token slots are four K steps of two sub-tiles.
// Gated: eight weight and five token slots are four K steps of gate and up.
struct FewRows { static constexpr int W = 7, X = 7; static constexpr bool GATED = false; };
struct ManyRows { static constexpr int W = 6, X = 8; static constexpr bool GATED = false; };
struct Gated { static constexpr int W = 8, X = 5; static constexpr bool GATED = true; };
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t ACC_COLS = 192;        // accumulators at columns [0,192) and [192,384)
constexpr uint32_t SF_COL0 = 384;         // per weight slot 16 columns: 4 (weight scales) + 12 (token scales)
constexpr uint32_t SF_SLOT_COLS = 16;
static_assert(SF_COL0 + Gated::W * SF_SLOT_COLS <= TMEM_COLS && FewRows::W <= Gated::W && ManyRows::W <= Gated::W, "TMEM budget");
static_assert(Gated::W % 2 == 0, "gate in the even slots, up in the odd ones");

constexpr int MAX_W = 8, MAX_X = 8;
constexpr uint32_t ERR_PRODUCER = 0x10u, ERR_MMA = 0x20u, ERR_EPILOGUE = 0x40u, ERR_SCHEDULER = 0x100u;
constexpr int W_WARP = 0, MMA_WARP = 1, SCHED_WARP = 2, X_WARP = 3, EPI_WARP0 = 4;
constexpr int EPI_WARPS = 12;                              // 4 TMEM lane quadrants x 3 warps
constexpr int EPI_BYTES_PER_WARP = 8 * 32 * 2;             // 8 tokens x 32 n
constexpr int QUEUE_DEPTH = 4;
// readers of a queue entry: both producers and the epilogue warps of each CTA, the MMA warp of the leader
constexpr int Q_CONSUMERS = 2 * (2 + EPI_WARPS) + 1;

struct Item {      // one work item as the scheduler hands it out
  int valid;       // token rows of the item (<= 384); -1: no more work
  int row0;        // first token row in a / d
  int n01;         // MMA N of the two sub-tiles, n0 | n1 << 16 (multiples of 16; n1 == 0: one sub-tile); gated: N | first
                   // column of the token scales in their atom << 16
  int np0;         // first weight pair
  int units;       // weight pairs of the item
  int e;           // expert
  int sfx_row;     // first 128-row block of the token scales
  int one_tile;    // 1: the expert has one token tile (its weights are read once)
};
static_assert(sizeof(Item) == 32, "two 16-byte words");

struct SharedCtl {
  uint64_t full[MAX_W];           // leader only: both producers' arrivals and all bytes of a K step
  uint64_t empty[MAX_W];          // the step's MMAs have completed: its weight slot and its token slots are free
  uint64_t acc_full[2];
  uint64_t acc_empty[2];          // leader only: one arrival per epilogue warp of both CTAs
  uint64_t q_full[QUEUE_DEPTH];
  uint64_t q_empty[QUEUE_DEPTH];  // leader only
  alignas(16) Item q_item[QUEUE_DEPTH];
  int x_user[MAX_X];              // token producer: the K step that used the slot last
  alignas(16) uint32_t tmem_base;
  int abort_flag;
  int warp_heavy[32], warp_light[32];
  int prefix_heavy[ES_B200_MAX_EXPERTS + 1];   // exclusive prefix of the experts' work items
  int prefix_light[ES_B200_MAX_EXPERTS + 1];
};

template <class S>
constexpr size_t smem_bytes() {
  return 1024 + (size_t)S::W * W_SLOT + (size_t)S::X * X_SLOT + EPI_WARPS * EPI_BYTES_PER_WARP + sizeof(SharedCtl);
}
static_assert(smem_bytes<FewRows>() <= 232448 && smem_bytes<ManyRows>() <= 232448 && smem_bytes<Gated>() <= 232448, "shared memory of one CTA per SM");

__device__ uint32_t g_status = 0;

struct Maps {
  CUtensorMap w;        // weights  [E*N, K] bytes, box 128 rows x 128 B, 128-byte swizzle
  CUtensorMap x[5];     // tokens   [T, K]   bytes, boxes of 8 / 16 / 32 / 64 / 96 rows
  CUtensorMap sfw;      // weight scale atoms, 512-byte records
  CUtensorMap sfx1;     // token scale atoms as [128-row block][K block] of 512-byte records; box = 1 row block
  CUtensorMap sfx3;     // the same, box = 3 row blocks
};

struct KernelArgs {
  void* d;                   // gated: the e4m3 codes
  uint8_t* scales;           // gated: their scale bytes
  const int* problem_sizes;
  const int* expert_offsets;
  const int* blockscale_offsets;
  int num_experts, n, k;     // n: weight rows per expert (gated: gate rows, as many up rows follow them)
  int heavy_min;             // experts with at least this many rows come first in the work list
  int group_heavy, group_light;   // weight pairs per work item
  uint32_t* counters;
};

__device__ __forceinline__ int box_index(int half_rows) {   // token tensor maps: boxes of 8 / 16 / 32 / 64 / 96 rows
  return half_rows <= 8 ? 0 : half_rows <= 16 ? 1 : half_rows <= 32 ? 2 : half_rows <= 64 ? 3 : 4;
}
__device__ __forceinline__ uint32_t box_rows_of(int idx) {
  return idx == 0 ? 8u : idx == 1 ? 16u : idx == 2 ? 32u : idx == 3 ? 64u : 96u;
}

// largest e in [0, n) with prefix[e] <= u, found by a converged warp (prefix non-decreasing, prefix[0] = 0 <= u < prefix[n])
__device__ __forceinline__ int warp_find_expert(const int* prefix, int n, int u, int lane) {
  const int stride = (n + 31) >> 5;
  const int i = lane * stride;
  const uint32_t above = __ballot_sync(0xffffffffu, i < n && prefix[i] <= u);
  const int lo = (31 - __clz((int)above)) * stride;
  const int j = lo + lane;
  const uint32_t in = __ballot_sync(0xffffffffu, lane < stride && j < n && prefix[j] <= u);
  return lo + 31 - __clz((int)in);
}

// 8 tokens per pass through the warp's shared-memory tile: held[4 g + b] is the 8x8 fragment (n 8b .. 8b+7, tokens
// 8g .. 8g+7) of a 32-token chunk; stored transposed, read back as 16-byte pieces of a token row, stored as 128-bit words,
// four lanes per 64-byte segment.  `tok`: first token of the chunk within the item.
template <typename OutT>
__device__ __forceinline__ void store_chunk_16B(const uint32_t (&held)[16], uint32_t stage, int tok, int valid, OutT* out,
                                                int64_t ld, int lane, bool scattered, OutT* dest_row) {
  const uint32_t wr = stage + (lane & 7) * 64 + (((lane >> 3) ^ ((lane & 7) >> 1)) << 4);
  const uint32_t rd = stage + (lane >> 2) * 64 + (((lane & 3) ^ ((lane >> 3) & 3)) << 4);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    if (tok + g * 8 >= valid) break;       // warp-uniform
    ptx::stmatrix_x4_trans(wr, held[g * 4], held[g * 4 + 1], held[g * 4 + 2], held[g * 4 + 3]);
    __syncwarp();
    const int t = g * 8 + (lane >> 2);
    const uint4 val = ptx::ld_shared_16B(rd);
    if (!scattered) {
      if (tok + t < valid) *reinterpret_cast<uint4*>(out + (int64_t)(tok + t) * ld + (lane & 3) * 8) = val;
    } else {
      OutT* row = reinterpret_cast<OutT*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(dest_row), t));
      if (row != nullptr) *reinterpret_cast<uint4*>(row + (lane & 3) * 8) = val;
    }
    __syncwarp();
  }
}

// 32-column chunks of the warp's 32 accumulator lanes as 16-bit 8x8 fragments (see store_chunk_16B): one chunk, or two with
// all four reads in flight
template <typename OutT>
__device__ __forceinline__ void pack_chunk(const uint32_t (&lo)[16], const uint32_t (&hi)[16], uint32_t (&held)[16]) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    held[4 * g + 0] = pack_pair_from_f32<OutT>(__uint_as_float(lo[4 * g]), __uint_as_float(lo[4 * g + 1]));
    held[4 * g + 1] = pack_pair_from_f32<OutT>(__uint_as_float(lo[4 * g + 2]), __uint_as_float(lo[4 * g + 3]));
    held[4 * g + 2] = pack_pair_from_f32<OutT>(__uint_as_float(hi[4 * g]), __uint_as_float(hi[4 * g + 1]));
    held[4 * g + 3] = pack_pair_from_f32<OutT>(__uint_as_float(hi[4 * g + 2]), __uint_as_float(hi[4 * g + 3]));
  }
}
// silu(g) * u in fp32 (hardware exponential and quotient: a few units in the last place, against 2^-4 of an e4m3 code)
__device__ __forceinline__ float silu_mul(float g, float u) { return __fdividef(g, 1.0f + __expf(-g)) * u; }

// gated: a chunk's fp32 fragments, and silu of them times the up accumulator's
__device__ __forceinline__ void read_fragments(uint32_t taddr, float (&v)[32]) {
  uint32_t lo[16], hi[16];
  ptx::tc_ld_16x256b_x4(taddr, lo);
  ptx::tc_ld_16x256b_x4(taddr + (16u << 16), hi);
  ptx::tc_wait_ld();
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = __uint_as_float(lo[i]);
    v[16 + i] = __uint_as_float(hi[i]);
  }
}
__device__ __forceinline__ void times_up(uint32_t taddr, float (&v)[32]) {
  uint32_t lo[16], hi[16];
  ptx::tc_ld_16x256b_x4(taddr, lo);
  ptx::tc_ld_16x256b_x4(taddr + (16u << 16), hi);
  ptx::tc_wait_ld();
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = silu_mul(v[i], __uint_as_float(lo[i]));
    v[16 + i] = silu_mul(v[16 + i], __uint_as_float(hi[i]));
  }
}
template <typename OutT>
__device__ __forceinline__ void read_chunk(uint32_t taddr, uint32_t (&held)[16]) {
  uint32_t lo[16], hi[16];
  ptx::tc_ld_16x256b_x4(taddr, lo);
  ptx::tc_ld_16x256b_x4(taddr + (16u << 16), hi);
  ptx::tc_wait_ld();
  pack_chunk<OutT>(lo, hi, held);
}
template <typename OutT>
__device__ __forceinline__ void read_two_chunks(uint32_t taddr0, uint32_t taddr1, uint32_t (&held0)[16], uint32_t (&held1)[16]) {
  uint32_t lo0[16], hi0[16], lo1[16], hi1[16];
  ptx::tc_ld_16x256b_x4(taddr0, lo0);
  ptx::tc_ld_16x256b_x4(taddr0 + (16u << 16), hi0);
  ptx::tc_ld_16x256b_x4(taddr1, lo1);
  ptx::tc_ld_16x256b_x4(taddr1 + (16u << 16), hi1);
  ptx::tc_wait_ld();
  pack_chunk<OutT>(lo0, hi0, held0);
  pack_chunk<OutT>(lo1, hi1, held1);
}

// Quantises a 32-token chunk of 32 outputs (one scale block per token) and stores codes and scale bytes.  v: fp32 fragments,
// v[4 g + 2 h + j] the value of output lane / 4 + 8 h, token 8 g + 2 (lane % 4) + j (h = 0, 1), v[16 + ...] the outputs 16
// further.  `codes`: first token, first output of the chunk; `scales`: the byte of token 0 of the item's atom rows and this
// block.  Arithmetic as in mxfp8_quant_math.cuh, from fp32 values.
__device__ __forceinline__ void store_chunk_quantised(const float (&v)[32], uint32_t stage, int tok, int valid, int sf_row,
                                                      uint8_t* codes, int64_t ld, uint8_t* scales, int kt_out, int lane) {
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    if (tok + p * 16 >= valid) break;       // warp-uniform
#pragma unroll
    for (int gl = 0; gl < 2; ++gl) {
      const int g = p * 2 + gl;
      float inv[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float m = fmaxf(fmaxf(fabsf(v[4 * g + j]), fabsf(v[4 * g + 2 + j])),
                        fmaxf(fabsf(v[16 + 4 * g + j]), fabsf(v[16 + 4 * g + 2 + j])));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        const uint32_t sf = __nv_cvt_float_to_e8m0(m * rcp_approx_ftz(448.0f), __NV_SATFINITE, cudaRoundPosInf);
        const uint32_t inv_bits = sf == 0 ? 0x7f800000u : sf == 255u ? 0x7fffffffu : (254u - sf) << 23;
        inv[j] = m != 0.f ? __uint_as_float(inv_bits) : 0.0f;
        const int t = tok + 8 * g + 2 * (lane & 3) + j;
        if ((lane >> 2) == g && t < valid) scales[scale_word_offset(sf_row + t, kt_out)] = (uint8_t)sf;
      }
      const uint32_t row = stage + (gl * 8 + 2 * (lane & 3)) * 32 + (lane >> 2);
#pragma unroll
      for (int h = 0; h < 4; ++h) {         // outputs lane / 4 + 8 h
        const int i = (h >> 1) * 16 + 4 * g + (h & 1) * 2;
        const uint32_t c = e4m3x4(make_float2(v[i] * inv[0], v[i + 1] * inv[1]), make_float2(0.f, 0.f));
        ptx::st_shared_u8(row + 8 * h, c);
        ptx::st_shared_u8(row + 32 + 8 * h, c >> 8);
      }
    }
    __syncwarp();
    const uint4 val = ptx::ld_shared_16B(stage + lane * 16);
    const int t = tok + p * 16 + (lane >> 1);
    if (t < valid) *reinterpret_cast<uint4*>(codes + (int64_t)(t - tok) * ld + (lane & 1) * 16) = val;
    __syncwarp();
  }
}

template <typename OutT, class S>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
mxfp8_grouped_mm_pair_kernel(const __grid_constant__ Maps maps, const __grid_constant__ KernelArgs args,
                             const __grid_constant__ RowScatter scatter) {
  constexpr int W_STAGES = S::W, X_STAGES = S::X;
  constexpr bool GATED = S::GATED;
  constexpr int TILE_ROWS = GATED ? SUB_TILE : 128 * ITEM_ATOMS;     // token rows of a work item at most
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = ptx::align1024(smem_raw);
  uint8_t* x_ring = smem + (size_t)W_STAGES * W_SLOT;
  uint8_t* epi_stage = x_ring + (size_t)X_STAGES * X_SLOT;
  SharedCtl* ctl = reinterpret_cast<SharedCtl*>(epi_stage + EPI_WARPS * EPI_BYTES_PER_WARP);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();      // 0 = leader (schedules, issues the MMAs), 1 = peer
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int num_experts = args.num_experts, n = args.n, k = args.k;

  if (threadIdx.x == SCHED_WARP * 32) {
    for (int s = 0; s < W_STAGES; ++s) {
      ptx::mbar_init(&ctl->full[s], GATED && (s & 1) ? 1 : 2);
      ptx::mbar_init(&ctl->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&ctl->acc_full[a], 1);
      ptx::mbar_init(&ctl->acc_empty[a], 2 * EPI_WARPS);
    }
    for (int q = 0; q < QUEUE_DEPTH; ++q) {
      ptx::mbar_init(&ctl->q_full[q], 1);
      ptx::mbar_init(&ctl->q_empty[q], Q_CONSUMERS);
    }
    ctl->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == MMA_WARP) {
    ptx::tmem_alloc_pair(&ctl->tmem_base, TMEM_COLS);
    ptx::tmem_relinquish_pair();
  }
  if (warp == W_WARP && lane < 9) {
    const CUtensorMap* m = lane == 0 ? &maps.w : lane < 6 ? &maps.x[lane - 1] : lane == 6 ? &maps.sfw : lane == 7 ? &maps.sfx1 : &maps.sfx3;
    ptx::prefetch_tensormap(m);
  }
  // (the wait for the partner's barriers is in the middle of the prologue: cluster_wait below)
  __syncthreads();
  ptx::cluster_arrive();
  pdl_wait_prior_grid();
  const int n_tiles = n / TILE_N;
  const int n_pairs = (n_tiles + 1) >> 1;
  const int kt_count = k / TILE_K;
  // rows, first row and first scale row of every expert, for the scheduler's first look-up: in the ring, which no load uses
  // before that
  int* const facts = reinterpret_cast<int*>(smem);
  if (rank == 0) {
    // exclusive prefixes of the experts' work items, heavy and light experts apart (an expert whose scales do not start
    // on a 128-row atom cannot be addressed: reported and skipped)
    const int per = (num_experts + THREADS - 1) / THREADS;      // 1 or 2 consecutive experts per thread
    const int heavy_groups = (n_pairs + args.group_heavy - 1) / args.group_heavy;
    const int light_groups = (n_pairs + args.group_light - 1) / args.group_light;
    int h[2] = {0, 0}, l[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = (int)threadIdx.x * per + i;
      if (i < per && e < num_experts) {
        const int m = args.problem_sizes[e * 3];
        const int bs = args.blockscale_offsets[e];
        facts[e] = m;
        facts[ES_B200_MAX_EXPERTS + e] = args.expert_offsets[e];
        facts[2 * ES_B200_MAX_EXPERTS + e] = bs;
        if (m > 0) {
          if ((bs & 127) != 0) atomicOr(&g_status, ERR_SCALE_OFFSET_BIT);
          else if (m >= args.heavy_min) h[i] = (int)(((int64_t)m + TILE_ROWS - 1) / TILE_ROWS) * heavy_groups;
          else l[i] = (int)(((int64_t)m + TILE_ROWS - 1) / TILE_ROWS) * light_groups;
        }
      }
    }
    int hs = h[0] + h[1], ls = l[0] + l[1];
#pragma unroll
    for (int dlt = 1; dlt < 32; dlt <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, hs, dlt), b = __shfl_up_sync(0xffffffffu, ls, dlt);
      if (lane >= dlt) { hs += a; ls += b; }
    }
    if (lane == 31) { ctl->warp_heavy[warp] = hs; ctl->warp_light[warp] = ls; }
    __syncthreads();
    int hb = 0, lb = 0;
    for (int w = 0; w < warp; ++w) { hb += ctl->warp_heavy[w]; lb += ctl->warp_light[w]; }
    hb += hs - h[0] - h[1];
    lb += ls - l[0] - l[1];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int e = (int)threadIdx.x * per + i;
      if (i < per && e < num_experts) {
        ctl->prefix_heavy[e] = hb;
        ctl->prefix_light[e] = lb;
        hb += h[i];
        lb += l[i];
      }
    }
    if (threadIdx.x == THREADS - 1) { ctl->prefix_heavy[num_experts] = hb; ctl->prefix_light[num_experts] = lb; }
  }
  // barriers, TMEM and prefixes must exist before either CTA signals the other
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_wait();
  ptx::tc_fence_after_sync();
  pdl_launch_dependents();

  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abort_flag = &ctl->abort_flag;
  int qs = 0;
  uint32_t qph = 0;
  // the next work item, read by a whole warp; false: a wait gave up
  auto next_item_one = [&](Item* it) {
    const bool have = rank == 0 ? ptx::mbar_wait(&ctl->q_full[qs], qph, abort_flag)
                                : ptx::mbar_wait_cluster(&ctl->q_full[qs], qph, abort_flag);
    if (!have) return false;
    const int4* src = reinterpret_cast<const int4*>(&ctl->q_item[qs]);
    *reinterpret_cast<int4*>(it) = src[0];
    *(reinterpret_cast<int4*>(it) + 1) = src[1];
    ptx::mbar_arrive_cluster_relaxed(&ctl->q_empty[qs], 0);
    if (++qs == QUEUE_DEPTH) { qs = 0; qph ^= 1u; }
    return true;
  };
  auto next_item = [&](Item* it) {
    const bool have = rank == 0 ? ptx::mbar_wait(&ctl->q_full[qs], qph, abort_flag)
                                : ptx::mbar_wait_cluster(&ctl->q_full[qs], qph, abort_flag);
    if (!__all_sync(0xffffffffu, have)) return false;
    const int4* src = reinterpret_cast<const int4*>(&ctl->q_item[qs]);
    *reinterpret_cast<int4*>(it) = src[0];
    *(reinterpret_cast<int4*>(it) + 1) = src[1];
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive_cluster_relaxed(&ctl->q_empty[qs], 0);
    if (++qs == QUEUE_DEPTH) { qs = 0; qph ^= 1u; }
    return true;
  };
  auto give_up = [&](uint32_t bit) {
    *abort_flag = 1;
    atomicOr(&g_status, bit);
  };

  if (warp == SCHED_WARP) {
    // ------------------------------------------------------------------ scheduler (leader): work item index -> item
    if (rank == 0) {
      const int total_heavy = ctl->prefix_heavy[num_experts], total = total_heavy + ctl->prefix_light[num_experts];
      // the first item of a pair is its own index, the counter deals the items from num_pairs on
      int t_next = pair;               // lane 0: the index that goes out next
      // The heavy items are dealt out evenly over the first 95 % of the list: next to one another they are bound by the
      // tensor pipe and the others by HBM (32768 Zipf rows, 256 experts, n = 4096, k = 7168: 1604 us with the heavy ones
      // first, 1521 so).  A long item must not be the last one.
      const bool mixed = total_heavy > 0 && total_heavy < total;
      const int64_t span = max((int64_t)total_heavy, (int64_t)total * 95 / 100);
      auto heavy_before = [&](int t) { return (int)min((int64_t)total_heavy, ((int64_t)t * total_heavy + span - 1) / span); };
      while (true) {
        const int t = __shfl_sync(0xffffffffu, t_next, 0);
        Item it = {-1, 0, 0, 0, 0, 0, 0, 0};
        if (t < total) {
          // the following index is requested now; its round trip to L2 hides behind this item
          if (lane == 0) t_next = args.counters ? num_pairs + (int)atomicAdd(args.counters, 1u) : t + num_pairs;
          bool heavy = total_heavy > 0;
          int u = t;
          if (mixed) {
            const int hb = heavy_before(t);
            heavy = heavy_before(t + 1) > hb;
            u = heavy ? hb : t - hb;
          }
          const int* prefix = heavy ? ctl->prefix_heavy : ctl->prefix_light;
          const int group = heavy ? args.group_heavy : args.group_light;
          const int e = warp_find_expert(prefix, num_experts, u, lane);
          const int i = u - prefix[e];
          const int m = t == pair ? facts[e] : args.problem_sizes[e * 3];
          const int row_first = t == pair ? facts[ES_B200_MAX_EXPERTS + e] : args.expert_offsets[e];
          const int sf_first = (t == pair ? facts[2 * ES_B200_MAX_EXPERTS + e] : args.blockscale_offsets[e]) >> 7;
          const int groups = (n_pairs + group - 1) / group;
          const int atoms = (m + 127) >> 7;
          const int tiles = (m + TILE_ROWS - 1) / TILE_ROWS;
          // Consecutive items run at the same time on different CTA pairs and share one operand in L2 while they sweep
          // the other: the swept operand should be the SMALLER one.
          int tt, g;
          if (tiles == 1) { tt = 0; g = i; }
          else if (m <= n) { g = i / tiles; tt = i - g * tiles; }
          else { tt = i / groups; g = i - tt * groups; }
          int first, rows, hi;
          if (GATED) {             // tiles of as many 64 rows as divide them evenly, 192 at most
            rows = (((m + tiles - 1) / tiles) + 63) & ~63;
            first = tt * rows;
            hi = (first >> 5) & 3;
          } else {                 // the atoms in tiles of base or base + 1
            const int base = atoms / tiles, rem = atoms - base * tiles;
            first = (tt * base + (tt < rem ? tt : rem)) * 128;
            rows = (base + (tt < rem ? 1 : 0)) * 128;
            hi = 0;
          }
          const int left = m - first;
          it.valid = left < rows ? left : rows;
          it.row0 = row_first + first;
          const int n0 = it.valid <= SUB_TILE ? (it.valid + 15) & ~15 : it.valid <= 256 ? 128 : SUB_TILE;
          if (!GATED) hi = it.valid > n0 ? (it.valid - n0 + 15) & ~15 : 0;
          it.n01 = n0 | (hi << 16);
          it.np0 = g * group;
          it.units = n_pairs - it.np0 < group ? n_pairs - it.np0 : group;
          it.e = e;
          it.sfx_row = sf_first + (first >> 7);
          it.one_tile = tiles == 1;
        }
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&ctl->q_empty[qs], qph ^ 1u, abort_flag))) {
          if (lane == 0) give_up(ERR_SCHEDULER);
          break;
        }
        if (t == pair) ptx::fence_proxy_async_shared();     // the facts have been read: loads may overwrite them
        if (lane == 0) {
          const int4 a = make_int4(it.valid, it.row0, it.n01, it.np0), b = make_int4(it.units, it.e, it.sfx_row, it.one_tile);
          int4* dst = reinterpret_cast<int4*>(&ctl->q_item[qs]);
          dst[0] = a;
          dst[1] = b;
          ptx::mbar_arrive(&ctl->q_full[qs]);
          ptx::send_32B_to_cluster_cta(&ctl->q_item[qs], &ctl->q_full[qs], 1, a, b);
        }
        __syncwarp();
        if (++qs == QUEUE_DEPTH) { qs = 0; qph ^= 1u; }
        if (it.valid < 0) break;
      }
    }
  } else if (warp == W_WARP) {
    // ------------------------------------------------------------------ weights and both scales of every K step (one thread)
    if (ptx::elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      while (ok) {
        Item it;
        ok = next_item_one(&it);
        if (!ok || it.valid < 0) break;
        const bool three = GATED || it.valid > 128;
        const uint32_t mine = W_BYTES + SF_BYTES + (three ? SFX_BYTES : SF_BYTES);
        const uint64_t hint = it.one_tile ? ptx::kL2EvictFirst : ptx::kL2EvictLast;
        const CUtensorMap* sfx_map = three ? &maps.sfx3 : &maps.sfx1;
        const int e_tile = it.e * n_tiles * (GATED ? 2 : 1);
        for (int u = 0; ok && u < it.units; ++u) {
          const int nt = (it.np0 + u) * 2 + (int)rank;
          const bool have = nt < n_tiles;          // n / 128 odd: the last pair's second half does not exist
          const uint32_t halves = (it.np0 + u) * 2 + 1 < n_tiles ? 2u : 1u;
          const int w_row = (e_tile + nt) * TILE_N;
          const int sfw_atom = (e_tile + nt) * kt_count;
          for (int kt = 0; kt < kt_count; ++kt) {
            ok = ptx::mbar_wait(&ctl->empty[s], ph ^ 1u, abort_flag);
            if (!ok) break;
            uint8_t* slot = smem + (size_t)s * W_SLOT;
            if (rank == 0) ptx::mbar_arrive_expect_tx(&ctl->full[s], mine * halves);
            if (have) {
              ptx::tma_load_2d_pair_hint(slot, &maps.w, &ctl->full[s], kt * TILE_K, w_row, hint);
              ptx::tma_load_2d_pair_hint(slot + W_BYTES, &maps.sfw, &ctl->full[s], 0, sfw_atom + kt, ptx::kL2EvictNormal);
              ptx::tma_load_2d_pair_hint(slot + W_BYTES + SF_BYTES, sfx_map, &ctl->full[s], kt * 128, it.sfx_row,
                                         ptx::kL2EvictNormal);
            }
            if (++s == W_STAGES) { s = 0; ph ^= 1u; }
            if constexpr (GATED) {                 // the up rows' slot (both slots of a step are freed together)
              ok = ptx::mbar_wait(&ctl->empty[s], ph ^ 1u, abort_flag);
              if (!ok) break;
              slot = smem + (size_t)s * W_SLOT;
              if (rank == 0) ptx::mbar_arrive_expect_tx(&ctl->full[s], (W_BYTES + SF_BYTES) * halves);
              if (have) {
                ptx::tma_load_2d_pair_hint(slot, &maps.w, &ctl->full[s], kt * TILE_K, w_row + n, hint);
                ptx::tma_load_2d_pair_hint(slot + W_BYTES, &maps.sfw, &ctl->full[s], 0, sfw_atom + n_tiles * kt_count + kt,
                                           ptx::kL2EvictNormal);
              }
              if (++s == W_STAGES) { s = 0; ph ^= 1u; }
            }
          }
        }
      }
      if (!ok) give_up(ERR_PRODUCER);
    }
    __syncwarp();
  } else if (warp == X_WARP) {
    // ------------------------------------------------------------------ token rows (one thread): one slot per sub-tile of a
    // K step.  A slot is free when the K step that used it last has completed, whose barrier is empty[] of that step's
    // weight slot.  A step further back than W_STAGES is not waited for but the one W_STAGES back is, whose weight slot this
    // step takes anyway: a parity wait cannot tell a phase from the one two further.
    if (ptx::elect_one()) {
      constexpr int PER_STEP = GATED ? 2 : 1, STEPS = W_STAGES / PER_STEP;     // weight slots per K step; K steps in the ring
      int s = 0, x = 0, step = 0;                     // s: weight slots of the step in K steps
      uint32_t ph = 0;
      for (int i = 0; i < X_STAGES; ++i) ctl->x_user[i] = -STEPS;
      bool ok = true;
      while (ok) {
        Item it;
        ok = next_item_one(&it);
        if (!ok || it.valid < 0) break;
        const int n0 = it.n01 & 0xffff, n1 = GATED ? 0 : it.n01 >> 16;
        const int xi0 = box_index(n0 >> 1), xi1 = box_index(n1 >> 1);
        const CUtensorMap* map0 = &maps.x[xi0];
        const CUtensorMap* map1 = &maps.x[xi1];
        const uint32_t tx = 2u * TILE_K * (box_rows_of(xi0) + (n1 ? box_rows_of(xi1) : 0u));
        const int row0 = it.row0 + (int)rank * (n0 >> 1), row1 = it.row0 + n0 + (int)rank * (n1 >> 1);
        for (int u = 0; ok && u < it.units; ++u) {
          for (int kt = 0; kt < kt_count; ++kt) {
            const int x1 = x + 1 == X_STAGES ? 0 : x + 1;
            int back = step - ctl->x_user[n1 ? x1 : x];      // the later of the slots' users, in steps back
            if (back > STEPS) back = STEPS;
            if (back <= step) {
              const int us = s - back;                       // its weight slot, of this revolution or of the one before
              ok = ptx::mbar_wait(&ctl->empty[(us < 0 ? us + STEPS : us) * PER_STEP + PER_STEP - 1], us < 0 ? ph ^ 1u : ph, abort_flag);
              if (!ok) break;
            }
            if (rank == 0) ptx::mbar_arrive_expect_tx(&ctl->full[s * PER_STEP], tx);
            ptx::tma_load_2d_pair_hint(x_ring + (size_t)x * X_SLOT, map0, &ctl->full[s * PER_STEP], kt * TILE_K, row0, ptx::kL2EvictLast);
            ctl->x_user[x] = step;
            x = x1;
            if (n1) {
              ptx::tma_load_2d_pair_hint(x_ring + (size_t)x * X_SLOT, map1, &ctl->full[s * PER_STEP], kt * TILE_K, row1, ptx::kL2EvictLast);
              ctl->x_user[x] = step;
              if (++x == X_STAGES) x = 0;
            }
            ++step;
            if (++s == STEPS) { s = 0; ph ^= 1u; }
          }
        }
      }
      if (!ok) give_up(ERR_PRODUCER);
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------------ scale copies and MMAs (leader, one thread)
    if (rank == 0 && ptx::elect_one()) {
      int s = 0, x = 0;
      uint32_t ph = 0, cnt = 0;
      const uint32_t smem_base = ptx::smem_u32(smem), x_base = ptx::smem_u32(x_ring);
      bool ok = true;
      while (ok) {
        Item it;
        ok = next_item_one(&it);
        if (!ok || it.valid < 0) break;
        // gated: both accumulators have the same token rows, the second one the up rows
        const int n0 = it.n01 & 0xffff, n1 = GATED ? n0 : it.n01 >> 16;
        const int sf_col = GATED ? it.n01 >> 16 : 0;      // first column of the token scales
        const int atoms = (it.valid + sf_col * 32 + 127) >> 7;
        const uint32_t idesc0 = ptx::make_idesc_mxf8(2 * TILE_N, n0, 0, 0), idesc1 = ptx::make_idesc_mxf8(2 * TILE_N, n1, 0, 0);
        for (int u = 0; ok && u < it.units; ++u) {
          const uint32_t a0 = cnt & 1u, a1 = a0 ^ 1u;
          ok = ptx::mbar_wait(&ctl->acc_empty[a0], ((cnt >> 1) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          // one K step's scale copies and MMAs of sub-tile 0
          auto first_half = [&](int kt) {
            if (!ptx::mbar_wait(&ctl->full[s], ph, abort_flag)) return false;
            ptx::tc_fence_after_sync();
            const uint32_t slot = smem_base + s * W_SLOT;
            const uint32_t sfw_t = tmem_base + SF_COL0 + s * SF_SLOT_COLS, sfx_t = sfw_t + 4;
            const uint64_t a_desc = ptx::make_desc_k_sw128(slot);
            const uint64_t sf_desc = ptx::make_desc_sf(slot + W_BYTES);
            const uint64_t b_desc = ptx::make_desc_k_sw128(x_base + x * X_SLOT);
            ptx::tc_cp_sf_pair(sfw_t, sf_desc);
            ptx::tc_cp_sf_pair(sfx_t, sf_desc + (512 >> 4));
            if (atoms > 1) ptx::tc_cp_sf_pair(sfx_t + 4, sf_desc + (1024 >> 4));
            if (atoms > 2) ptx::tc_cp_sf_pair(sfx_t + 8, sf_desc + (1536 >> 4));
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
              ptx::tc_mma_mxf8_pair(tmem_base + a0 * ACC_COLS, a_desc + 2 * j, b_desc + 2 * j, idesc0 | (j << 4) | (j << 29),
                                    sfw_t | (j << 30), (sfx_t + sf_col) | (j << 30), (kt | j) != 0 ? 1u : 0u);
            return true;
          };
          // the MMAs of sub-tile 1 of the K step in weight slot sl, token slot xl (gated: of the up rows, in the slot behind)
          auto second_half = [&](int kt, int sl, int xl, uint32_t phl) {
            const int wl = GATED ? sl + 1 : sl;
            if (GATED) {
              if (!ptx::mbar_wait(&ctl->full[wl], phl, abort_flag)) return false;
              ptx::tc_fence_after_sync();
              ptx::tc_cp_sf_pair(tmem_base + SF_COL0 + wl * SF_SLOT_COLS, ptx::make_desc_sf(smem_base + wl * W_SLOT + W_BYTES));
            }
            const uint32_t sfw_t = tmem_base + SF_COL0 + wl * SF_SLOT_COLS;
            // sub-tile 1 starts n0 rows into the token scales
            const uint32_t sfx_t = tmem_base + SF_COL0 + sl * SF_SLOT_COLS + 4 + (GATED ? sf_col : n0 >> 5);
            const uint64_t a_desc = ptx::make_desc_k_sw128(smem_base + wl * W_SLOT);
            const uint64_t b_desc = ptx::make_desc_k_sw128(x_base + xl * X_SLOT);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
              ptx::tc_mma_mxf8_pair(tmem_base + a1 * ACC_COLS, a_desc + 2 * j, b_desc + 2 * j, idesc1 | (j << 4) | (j << 29),
                                    sfw_t | (j << 30), sfx_t | (j << 30), (kt | j) != 0 ? 1u : 0u);
            ptx::tc_commit_pair(&ctl->empty[sl], 3);
            if (GATED) ptx::tc_commit_pair(&ctl->empty[wl], 3);
            return true;
          };
          auto next_x = [&](int i) { return i + 1 == X_STAGES ? 0 : i + 1; };
          auto next_step = [&]() { if ((s += GATED ? 2 : 1) == W_STAGES) { s = 0; ph ^= 1u; } };
          if (n1 == 0) {
            for (int kt = 0; ok && kt < kt_count; ++kt) {
              ok = first_half(kt);
              if (!ok) break;
              ptx::tc_commit_pair(&ctl->empty[s], 3);
              x = next_x(x);
              next_step();
            }
            if (!ok) break;
            ptx::tc_commit_pair(&ctl->acc_full[a0], 3);
            cnt += 1;
          } else {
            // The first two and the last two K steps go sub-tile by sub-tile: accumulator 0 is then complete 2 x 4 MMAs before
            // accumulator 1 and wanted back as much earlier, which hides the time that the epilogue takes to empty it.
            for (int kt = 0; ok && kt < kt_count;) {
              const bool two = kt + 1 < kt_count && (kt == 0 || kt + 2 == kt_count);
              // (gated: gate and up multiply the same token slot)
              const int s0 = s, x0 = GATED ? x : next_x(x);
              const uint32_t ph0 = ph;
              ok = first_half(kt);
              if (!ok) break;
              x = next_x(x0);
              next_step();
              const int s1 = s;
              const uint32_t ph1 = ph;
              int x1 = 0;
              if (two) {
                x1 = GATED ? x : next_x(x);
                ok = first_half(kt + 1);
                if (!ok) break;
                x = next_x(x1);
                next_step();
              }
              if (kt + (two ? 2 : 1) == kt_count) ptx::tc_commit_pair(&ctl->acc_full[a0], 3);
              if (kt == 0) {
                ok = ptx::mbar_wait(&ctl->acc_empty[a1], (((cnt + 1) >> 1) & 1u) ^ 1u, abort_flag);
                if (!ok) break;
                ptx::tc_fence_after_sync();
              }
              ok = second_half(kt, s0, x0, ph0) && (!two || second_half(kt + 1, s1, x1, ph1));
              if (!ok) break;
              kt += two ? 2 : 1;
            }
            if (!ok) break;
            ptx::tc_commit_pair(&ctl->acc_full[a1], 3);
            cnt += 2;
          }
        }
      }
      if (!ok) give_up(ERR_MMA);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue (both CTAs), 12 warps: three per TMEM lane
    // quadrant share the 32-column chunks of the accumulators, at most two per sub-tile.  A warp reads its chunks of a
    // weight pair's accumulators into registers (converted), hands each accumulator back, and stores afterwards: the next
    // weight pair's MMAs run during the stores.
    const int q = warp & 3;
    const int idx = (warp - EPI_WARP0) >> 2;      // 0..2 within the lane quadrant
    const uint32_t stage = ptx::smem_u32(epi_stage) + (warp - EPI_WARP0) * EPI_BYTES_PER_WARP;
    const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
    OutT* const d = static_cast<OutT*>(args.d);
    const bool scattered = scatter.meta != nullptr;
    uint32_t cnt = 0;
    int turn = idx;                               // first chunk of this warp; rotates so that small tiles go round
    bool ok = true;
    while (ok) {
      Item it;
      ok = next_item(&it);
      if (!ok || it.valid < 0) break;
      const int n0 = it.n01 & 0xffff, n1 = GATED ? n0 : it.n01 >> 16;
      for (int u = 0; u < it.units; ++u) {
        const int nt = (it.np0 + u) * 2 + (int)rank;
        const int col_off = nt * TILE_N + q * 32;
        const uint32_t a0 = cnt & 1u, a1 = a0 ^ 1u;
        const uint32_t p0 = (cnt >> 1) & 1u, p1 = ((cnt + 1) >> 1) & 1u;
        const int c0 = turn * 32, c1 = c0 + 96;
        if constexpr (GATED) {
          // this warp's chunks of the gate accumulator, then each one's up values: silu(gate) * up in their place
          float act0[32], act1[32];
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->acc_full[a0], p0, abort_flag));
          if (!ok) break;
          ptx::tc_fence_after_sync();
          const uint32_t t0 = lane_base + a0 * ACC_COLS, t1 = lane_base + a1 * ACC_COLS;
          if (c0 < n0) read_fragments(t0 + c0, act0);
          if (c1 < n0) read_fragments(t0 + c1, act1);
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster_relaxed(&ctl->acc_empty[a0], 0);
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->acc_full[a1], p1, abort_flag));
          if (!ok) break;
          ptx::tc_fence_after_sync();
          if (c0 < n0) times_up(t1 + c0, act0);
          if (c1 < n0) times_up(t1 + c1, act1);
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster_relaxed(&ctl->acc_empty[a1], 0);
          if (nt < n_tiles) {
            // scale block of these 32 outputs: K block col_off / 32 of the next GEMM's operand
            uint8_t* codes = static_cast<uint8_t*>(args.d) + (int64_t)it.row0 * n + col_off;
            uint8_t* scales = args.scales + ((int64_t)it.sfx_row * n_tiles + nt) * 512 + q;
            const int sf_row = (it.n01 >> 16) * 32;
            if (c0 < n0) store_chunk_quantised(act0, stage, c0, it.valid, sf_row, codes + (int64_t)c0 * n, n, scales, n_tiles, lane);
            if (c1 < n0) store_chunk_quantised(act1, stage, c1, it.valid, sf_row, codes + (int64_t)c1 * n, n, scales, n_tiles, lane);
          }
          cnt += 2;
          turn = turn == 0 ? 2 : turn - 1;
          continue;
        }
        uint32_t held[4][16];
        ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->acc_full[a0], p0, abort_flag));
        if (!ok) break;
        ptx::tc_fence_after_sync();
        const uint32_t t0 = lane_base + a0 * ACC_COLS, t1 = lane_base + a1 * ACC_COLS;
        if (c1 < n0) read_two_chunks<OutT>(t0 + c0, t0 + c1, held[0], held[1]);
        else if (c0 < n0) read_chunk<OutT>(t0 + c0, held[0]);
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster_relaxed(&ctl->acc_empty[a0], 0);
        if (n1 != 0) {
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(&ctl->acc_full[a1], p1, abort_flag));
          if (!ok) break;
          ptx::tc_fence_after_sync();
          if (c0 < n1) read_chunk<OutT>(t1 + c0, held[2]);
          if (c1 < n1) read_chunk<OutT>(t1 + c1, held[3]);
          ptx::tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster_relaxed(&ctl->acc_empty[a1], 0);
        }
        if (nt < n_tiles) {
          OutT* out = d + (int64_t)it.row0 * n + col_off;
          auto store = [&](const uint32_t (&h)[16], int tok) {
            OutT* dest = nullptr;
            if (scattered)
              dest = scatter_row_ptr<OutT>(scatter, it.row0 + tok + lane, tok + lane < it.valid, n, col_off, &g_status);
            store_chunk_16B<OutT>(h, stage, tok, it.valid, out, n, lane, scattered, dest);
          };
          if (c0 < n0) store(held[0], c0);
          if (c1 < n0) store(held[1], c1);
          if (c0 < n1) store(held[2], n0 + c0);
          if (c1 < n1) store(held[3], n0 + c1);
        }
        cnt += n1 != 0 ? 2 : 1;
        turn = turn == 0 ? 2 : turn - 1;
      }
    }
    if (!ok && lane == 0) give_up(ERR_EPILOGUE);
  }

  if (scatter.meta != nullptr) __threadfence_system();
  // neither CTA may leave (or free TMEM) while its partner can still signal it or read its shared memory
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::settle_if_aborted(abort_flag);
  ptx::cluster_sync();
  if (warp == MMA_WARP) {
    __syncwarp();
    ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
  // the last CTA of the call clears the counters
  if (threadIdx.x == 0 && args.counters != nullptr && atomicAdd(&args.counters[1], 1u) == gridDim.x - 1) {
    args.counters[0] = 0;
    args.counters[1] = 0;
  }
}

template <typename OutT, class S>
int launch_as(const CallArgs& c) {
  DeviceInfo info;
  int rc = get_device_info(&info);
  if (rc != ES_B200_OK) return rc;
  const int kt_count = c.k / TILE_K;

  Maps maps;
  const uint64_t w_rows = (uint64_t)c.num_experts * c.n * (S::GATED ? 2 : 1);
  rc = make_tensormap_u8_sw128(&maps.w, c.b, w_rows, (uint64_t)c.k, TILE_N);
  if (rc != ES_B200_OK) return rc;
  const uint32_t boxes[5] = {8, 16, 32, 64, 96};
  for (int i = 0; i < 5; ++i) {
    rc = make_tensormap_u8_sw128(&maps.x[i], c.a, (uint64_t)c.num_rows, (uint64_t)c.k, boxes[i]);
    if (rc != ES_B200_OK) return rc;
  }
  rc = make_tensormap_records512(&maps.sfw, c.sfb, w_rows / TILE_N * kt_count);
  if (rc != ES_B200_OK) return rc;
  // whole 128-row atoms only; loads past the end read as zero (a map needs at least one row)
  const uint64_t sfx_rows = (uint64_t)(c.sfa_rows / 128);
  rc = make_tensormap_record_columns(&maps.sfx1, c.sfa, sfx_rows ? sfx_rows : 1, (uint64_t)kt_count, 1);
  if (rc != ES_B200_OK) return rc;
  rc = make_tensormap_record_columns(&maps.sfx3, c.sfa, sfx_rows ? sfx_rows : 1, (uint64_t)kt_count, ITEM_ATOMS);
  if (rc != ES_B200_OK) return rc;

  auto kernel = mxfp8_grouped_mm_pair_kernel<OutT, S>;
  static bool configured[64] = {false};
  static int resident_pairs[64] = {0};
  int dev = 0;
  ES_CUDA_TRY(cudaGetDevice(&dev));
  if (!configured[dev & 63]) {
    ES_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<S>()));
    configured[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem_bytes<S>();
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1] = c.overlap;
  cfg.attrs = attr;
  cfg.numAttrs = 1;

  // how many CTA pairs can be resident at once (SMs pair up inside a GPC, so this can be below sm_count / 2)
  if (resident_pairs[dev & 63] == 0) {
    cfg.gridDim = dim3(info.sm_count & ~1);
    int nc = 0;
    ES_CUDA_TRY(cudaOccupancyMaxActiveClusters(&nc, kernel, &cfg));
    if (nc < 1) return fail(ES_B200_ERR_CUDA, "no CTA pair of the grouped GEMM kernel fits on this device");
    resident_pairs[dev & 63] = nc;
  }
  if (attr[1].id == cudaLaunchAttributeProgrammaticStreamSerialization) cfg.numAttrs = 2;
  const int n_pairs = (c.n / TILE_N + 1) / 2;
  const int64_t used = c.num_experts < c.num_rows ? c.num_experts : c.num_rows;
  const int most_light = weight_tiles_per_item(tunables().mm_item_k_steps, kt_count * (S::GATED ? 2 : 1),
                                               used * n_pairs, info.sm_count);
  const int light_items = (n_pairs + most_light - 1) / most_light;
  const int group_light = (n_pairs + light_items - 1) / light_items;     // all of about the same length
  const int group_heavy = (group_light + 3) / 4;
  const int tile_rows = S::GATED ? SUB_TILE : 128 * ITEM_ATOMS;
  const int64_t max_items = ((c.num_rows + tile_rows - 1) / tile_rows + c.num_experts) * (int64_t)n_pairs;
  int max_pairs = resident_pairs[dev & 63];
  if (c.max_pairs > 0 && c.max_pairs < max_pairs) max_pairs = c.max_pairs;
  cfg.gridDim = dim3(2 * (unsigned)(max_items < max_pairs ? max_items : max_pairs));
  KernelArgs args = {c.d, c.scales, c.ps, c.eo, c.bo, c.num_experts, c.n, c.k, c.heavy_min, group_heavy, group_light, c.counters};
  ES_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, maps, args, *c.scatter));
  return ES_B200_OK;
}

// Which division of shared memory, by the mean number of rows per expert (the only thing about them that the host knows):
// 512 rows on 256 experts, n = 7168, k = 2048 239 us with seven weight slots, 246 with six; 64 experts of 100 rows, n = k =
// 2048 55.4 and 56.5; 256 rows on each of 128 experts, n = 1536, k = 2048 128.5 and 117.6; 32768 Zipf rows on 256 experts,
// n = 4096, k = 7168 1604 and 1589; 14600 rows of 1 to 1000 on 256 experts, n = 7168, k = 256 125.0 and 123.1.
template <typename OutT>
int launch(const CallArgs& c) {
  return c.num_rows < (int64_t)112 * c.num_experts ? launch_as<OutT, FewRows>(c) : launch_as<OutT, ManyRows>(c);
}
int launch_bf16(const CallArgs& c) { return launch<__nv_bfloat16>(c); }
int launch_fp16(const CallArgs& c) { return launch<__half>(c); }
int launch_silu_mul_quant(const CallArgs& c) { return launch_as<__nv_bfloat16, Gated>(c); }

int read_and_clear_status(uint32_t* out) {
  uint32_t v = 0;
  ES_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_status, sizeof(v)));
  if (v != 0) {
    uint32_t zero = 0;
    ES_CUDA_TRY(cudaMemcpyToSymbol(g_status, &zero, sizeof(zero)));
  }
  *out = v;
  return ES_B200_OK;
}

}  // namespace mm
}  // namespace es_b200
