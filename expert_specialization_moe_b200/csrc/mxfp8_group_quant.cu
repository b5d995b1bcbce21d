// MXFP8 grouped quantisation for sm_100a: bf16/fp16 rows -> e4m3 codes + UE8M0 scale per 32 elements, scales
// written straight into the SM100 swizzled layout (512-byte atoms of 128 rows x 4 K-blocks) at per-expert offsets.
//
// Arithmetic contract (bit-exact with the reference kernel, es_sm100_mxfp8_blockscaled_group_quant.cuh:36-134):
//   amax  = max |x_i| over the 32-block, NaN members dropped (max.bf16x2 / max.f16x2 semantics)
//   s     = fp32(amax) * rcp.approx.ftz.f32(448.0f)
//   sf    = cvt.rp.satfinite.ue8m0x2.f32(s)
//   inv   = amax != 0 ? rcp.approx.ftz.f32(float(sf)) : 0
//   code  = cvt.rn.satfinite.e4m3x2.f32(fp32(x_i) * inv)
//
// Schedule: an expert's rows are one contiguous stream of 128-element K tiles (rows are densely packed), whatever k is.
// Eight lanes take a tile, sixteen elements each; a warp takes four consecutive tiles per step and `steps` steps per
// work unit.  Units of all experts form one flat list found with a per-CTA prefix scan over the row counts, so neither
// the split of the rows between experts nor k leaves lanes idle, and a call of a few rows is spread over as many warps
// as it has tiles (the host picks `steps` from the row count).  Zeroing the scale bytes of the padding rows is work
// units of its own, in 16-byte pieces: in a decode call they are as many bytes as the codes.
//
// What bounds it: HBM (3 + 1/32 bytes per element; with silu 5 + 1/32).  One lane per 8 elements and a warp per row
// cost 10.5 instructions per element, enough to keep the issue slots 62 % busy; 16 elements per lane halve the scale
// arithmetic, shuffles and addresses per element.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <type_traits>

#include "common.cuh"
#include "mxfp8_quant_math.cuh"

namespace es_b200 {

constexpr int QUANT_THREADS = 256;
constexpr int QUANT_WARPS = QUANT_THREADS / 32;
constexpr int QUANT_TILES_PER_STEP = 4;       // a warp's four groups of eight lanes, one 128-element K tile each
constexpr int QUANT_PAD_ATOMS = 16;           // scale atoms per unit of padding work
constexpr int QUANT_MAX_STEPS_LOG2 = 4;
// registers: two steps of input in flight per warp; the fused variant holds gate and up of both
constexpr int QUANT_MIN_BLOCKS = 4, QUANT_MIN_BLOCKS_SILU = 3;

// exact arithmetic of an unfused silu(gate.float()) * up.float() -> T: accurate expf, IEEE division and multiply
__device__ __forceinline__ float silu_mul_exact(float g, float u) { return (g / (1.0f + expf(-g))) * u; }

// act = round_to_T( silu(gate) * up ) on two elements, bit for bit what silu_mul_exact gives, for a quarter of its
// instructions: p = g * rcp(1 + 2^(-g log2 e)) * u with the hardware approximations is within `eps` (relative) of the
// exact sequence's fp32 value, so wherever p (1 - eps) and p (1 + eps) round to the same 16-bit value, that value is the
// answer (rounding is monotonic); the few pairs where they do not (bf16: 0.04 % of the elements) take the exact
// sequence.  `wild` sends a pair there too: |g| > 64, where 1 + 2^x can leave the range of the approximate reciprocal.
// Error of p against the exact sequence, in units of 2^-24: 2^x 4 (2 ulp), its argument |g| (one rounding of g log2 e
// and of the constant), reciprocal 2 (1 ulp), sum and two products 3 x 1; exact sequence: expf 2 (1 ulp), sum, quotient
// and product 3 x 1; rounding of the two bounds 2.  16 + |g| in all; eps = (24 + 1.5 |g|) 2^-24.
// bf16 gates and results below 2^-100 (zeros among them) also go the exact way: the bounds are relative, and next to
// the fp32 subnormals a relative bound says nothing.  fp16 values are at least 2^-24, so q and p cannot get there.
template <typename T>
__device__ __forceinline__ uint32_t silu_mul2(uint32_t gw, uint32_t uw, float eps, bool wild) {
  using V2 = typename Vec2<T>::type;
  const float2 g = Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&gw));
  const float2 u = Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&uw));
  const float2 t = mul2(g, make_float2(-1.4426950408889634f, -1.4426950408889634f));
  const float2 d = add2(make_float2(ex2_approx_ftz(t.x), ex2_approx_ftz(t.y)), make_float2(1.0f, 1.0f));
  const float2 q = mul2(g, make_float2(rcp_approx_ftz(d.x), rcp_approx_ftz(d.y)));
  const float2 p = mul2(q, u);
  const float2 hi = fma2(p, make_float2(eps, eps), p);
  const float2 lo = fma2(p, make_float2(-eps, -eps), p);
  V2 r = Vec2<T>::from_floats(hi.x, hi.y);
  const V2 r2 = Vec2<T>::from_floats(lo.x, lo.y);
  uint32_t out = *reinterpret_cast<const uint32_t*>(&r);
  uint32_t differ = out ^ *reinterpret_cast<const uint32_t*>(&r2);
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    const uint32_t limit = 0x0d800d80u;      // 2^-100 twice
    differ |= __hlt2_mask(__habs2(r), *reinterpret_cast<const V2*>(&limit)) |
              __hlt2_mask(__habs2(*reinterpret_cast<const V2*>(&gw)), *reinterpret_cast<const V2*>(&limit));
  }
  if (differ != 0 || wild) {
    r = Vec2<T>::from_floats(silu_mul_exact(g.x, u.x), silu_mul_exact(g.y, u.y));
    out = *reinterpret_cast<const uint32_t*>(&r);
  }
  return out;
}

// 32 bytes of input per lane: one 256-bit load where the tensor starts on a 32-byte boundary (tiles are multiples of
// 256 bytes), two 128-bit loads otherwise
template <bool kWide>
__device__ __forceinline__ void load_16_elements(const void* p, uint32_t (&v)[8]) {
  if constexpr (kWide) {
    ld_stream_32B(p, v);
  } else {
    const uint4 a = ld_stream_16B(p), b = ld_stream_16B(static_cast<const uint8_t*>(p) + 16);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
}

// kSiluMul = false: input [rows, k].  kSiluMul = true: input [rows, 2k] = gate | up, quantises silu(gate) * up.
template <typename T, bool kSiluMul, bool kWide>
__global__ void __launch_bounds__(QUANT_THREADS, kSiluMul ? QUANT_MIN_BLOCKS_SILU : QUANT_MIN_BLOCKS)
mxfp8_group_quant_kernel(const T* __restrict__ input, const int* __restrict__ problem_sizes,
                         const int* __restrict__ expert_offsets, const int* __restrict__ blockscale_offsets,
                         uint8_t* __restrict__ quant_output, uint8_t* __restrict__ scale_factor, int num_experts,
                         int k, int steps_log2) {
  __shared__ int table[ES_B200_MAX_EXPERTS + 1];
  __shared__ int warp_sums[32];

  const int kt = k >> 7;                          // K tiles (= 32-bit scale words) per row
  const int unit_log2 = 2 + steps_log2;           // tiles per unit, as a power of two
  const int pad_units = (kt + QUANT_PAD_ATOMS - 1) / QUANT_PAD_ATOMS;
  // (a tile is at least 256 bytes of input: 32 bits count the tiles of any tensor that fits the GPU)
  auto data_units = [&](int m) { return (int)(((uint32_t)m * (uint32_t)kt + (1u << unit_log2) - 1u) >> unit_log2); };
  pdl_wait_prior_grid();
  block_exclusive_scan(num_experts, table, warp_sums, [&](int e) {
    const int m = problem_sizes[e * 3];
    return m > 0 ? data_units(m) + ((m & 127) ? pad_units : 0) : 0;
  });
  const ExpertTable tab = fill_expert_table(table, num_experts, problem_sizes, expert_offsets, blockscale_offsets);
  __syncthreads();
  pdl_launch_dependents();
  const int total_units = table[num_experts];

  const int lane = threadIdx.x & 31;
  const int group = lane >> 3, l8 = lane & 7;     // this lane's tile of the step, and its 16 elements of the tile

  // neighbouring units on neighbouring SMs first: a call of few units is spread over the whole GPU
  for (int u = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < total_units; u += gridDim.x * QUANT_WARPS) {
    const int e = upper_bound_expert(tab.prefix, num_experts, u);
    const int i = u - tab.prefix[e];
    const int m = tab.m(e);
    uint8_t* sf_expert = scale_factor + (int64_t)tab.scale0(e) * (k >> 5);
    const int n_data = data_units(m);
    if (i >= n_data) {
      // scale bytes of the padding rows m .. align128(m) - 1: lane j clears, in each atom, the words of its line (rows
      // j, j + 32, j + 64, j + 96 of the last 128) that belong to rows past the end
      const int last = m & 127;
      const int first_word = last <= lane ? 0 : (last - lane + 31) >> 5;      // 0 .. 4
      uint8_t* line = sf_expert + (int64_t)(m >> 7) * kt * 512 + lane * 16;
      const int q_end = min(kt, (i - n_data + 1) * QUANT_PAD_ATOMS);
      for (int q = (i - n_data) * QUANT_PAD_ATOMS; q < q_end; ++q) {
        uint32_t* words = reinterpret_cast<uint32_t*>(line + (int64_t)q * 512);
        if (first_word == 0 && (reinterpret_cast<uintptr_t>(words) & 15u) == 0) {
          *reinterpret_cast<uint4*>(words) = make_uint4(0, 0, 0, 0);
        } else {
          for (int w = first_word; w < 4; ++w) words[w] = 0u;
        }
      }
      continue;
    }
    const uint32_t t0 = ((uint32_t)i << unit_log2) + (uint32_t)group;               // this lane group's first tile
    const int tiles_left = (int)((uint32_t)m * (uint32_t)kt - ((uint32_t)i << unit_log2));   // from the unit's first on
    const int n_steps = min(1 << steps_log2, (tiles_left + QUANT_TILES_PER_STEP - 1) / QUANT_TILES_PER_STEP);
    int row = (int)(t0 / (uint32_t)kt);
    int q = (int)(t0 - (uint32_t)row * (uint32_t)kt);
    int load_row = row, load_q = q;
    const int64_t row0 = tab.row0(e);
    const T* src = input + row0 * (kSiluMul ? 2 * (int64_t)k : (int64_t)k) + l8 * 16;
    uint8_t* dst = quant_output + (row0 * kt + t0) * 128 + l8 * 16;

    uint32_t raw[2][8], raw_up[kSiluMul ? 2 : 1][8];
    auto load = [&](int s, uint32_t (&g)[8], uint32_t (&up)[8]) {
      if (s < n_steps && s * QUANT_TILES_PER_STEP + group < tiles_left) {
        if constexpr (kSiluMul) {
          const T* p = src + ((int64_t)load_row * 2 * kt + load_q) * 128;
          load_16_elements<kWide>(p, g);
          load_16_elements<kWide>(p + k, up);
          load_q += QUANT_TILES_PER_STEP;
          while (load_q >= kt) { load_q -= kt; ++load_row; }
        } else {
          load_16_elements<kWide>(src + ((int64_t)t0 + s * QUANT_TILES_PER_STEP) * 128, g);
        }
      }
    };
    auto step = [&](int s, uint32_t (&g)[8], uint32_t (&up)[8]) {
      uint32_t v[8];
      if constexpr (kSiluMul) {
        const float g_max = max_abs16<T>(g);
        const bool wild = !(g_max <= 64.0f);
        const float eps = fmaf(g_max, 8.940696716e-8f, 1.430511475e-6f);      // (24 + 1.5 |g|) 2^-24
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = silu_mul2<T>(g[j], up[j], eps, wild);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = g[j];
      }
      load(s + 2, g, up);
      uint4 codes;
      const uint32_t sf = quantize16<T>(v, codes);
      // the four scale bytes of the tile as one aligned 32-bit word (two lanes hold the byte of a 32-element block)
      uint32_t w = sf << ((l8 >> 1) * 8);
      w |= __shfl_xor_sync(0xffffffffu, w, 2);
      w |= __shfl_xor_sync(0xffffffffu, w, 4);
      if (s * QUANT_TILES_PER_STEP + group < tiles_left) {
        st_stream_16B(dst + (int64_t)s * (QUANT_TILES_PER_STEP * 128), codes);
        if (l8 == 0) *reinterpret_cast<uint32_t*>(sf_expert + scale_word_offset(row, kt) + (int64_t)q * 512) = w;
      }
      q += QUANT_TILES_PER_STEP;
      while (q >= kt) { q -= kt; ++row; }
    };
#pragma unroll
    for (int b = 0; b < 2; ++b) {
#pragma unroll
      for (int j = 0; j < 8; ++j) raw[b][j] = 0u;      // tiles past the end quantise zeros and store nothing
      if constexpr (kSiluMul) {
#pragma unroll
        for (int j = 0; j < 8; ++j) raw_up[b][j] = 0u;
      }
    }
    load(0, raw[0], raw_up[0]);
    load(1, raw[1], raw_up[kSiluMul ? 1 : 0]);
    for (int s = 0; s < n_steps; s += 2) {
      step(s, raw[0], raw_up[0]);
      if (s + 1 < n_steps) step(s + 1, raw[1], raw_up[kSiluMul ? 1 : 0]);
    }
  }
}

template <typename T, bool kSiluMul, bool kWide>
static int launch_quant(const void* input, const int32_t* problem_sizes, const int32_t* expert_offsets,
                        const int32_t* blockscale_offsets, void* quant_output, uint8_t* scale_factor, int num_experts,
                        int64_t num_rows, int k, cudaStream_t stream) {
  DeviceInfo info;
  int rc = get_device_info(&info);
  if (rc != ES_B200_OK) return rc;
  auto kernel = mxfp8_group_quant_kernel<T, kSiluMul, kWide>;
  static int blocks_per_sm = 0;      // same on every device of a box
  if (blocks_per_sm == 0) {
    int v = 0;
    ES_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, QUANT_THREADS, 0));
    blocks_per_sm = v > 0 ? v : 1;
  }
  const int64_t resident = (int64_t)info.sm_count * blocks_per_sm;
  // steps per unit: as many as leave every resident warp about four units (a short tail), 16 at most
  const int kt = k >> 7;
  const int64_t steps_total = (num_rows * kt + QUANT_TILES_PER_STEP - 1) / QUANT_TILES_PER_STEP;
  int steps_log2 = 0;
  while (steps_log2 < QUANT_MAX_STEPS_LOG2 && (steps_total >> (steps_log2 + 1)) >= 4 * resident * QUANT_WARPS) ++steps_log2;
  // at most one partial unit and the padding units per expert on top of the full units of num_rows rows
  const int64_t max_units = (steps_total >> steps_log2) + 1 +
                            (int64_t)num_experts * (1 + (kt + QUANT_PAD_ATOMS - 1) / QUANT_PAD_ATOMS);
  const int64_t max_ctas = (max_units + QUANT_WARPS - 1) / QUANT_WARPS;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(max_ctas < resident ? max_ctas : resident));
  cfg.blockDim = dim3(QUANT_THREADS);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ES_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<const T*>(input), problem_sizes, expert_offsets,
                                 blockscale_offsets, static_cast<uint8_t*>(quant_output), scale_factor, num_experts, k,
                                 steps_log2));
  return ES_B200_OK;
}

template <bool kSiluMul>
static int quant_impl(const void* input, int input_dtype, const int32_t* problem_sizes, const int32_t* expert_offsets,
                      const int32_t* blockscale_offsets, void* quant_output, uint8_t* scale_factor, int num_experts,
                      int64_t num_rows, int k, void* stream) {
  ES_REQUIRE(input_dtype == ES_B200_BF16 || input_dtype == ES_B200_FP16, "dtype must be kFloat16 or kBFloat16");
  ES_REQUIRE(k > 0 && k % 128 == 0, "k must align to 128");
  ES_REQUIRE(num_experts >= 0 && num_experts <= ES_B200_MAX_EXPERTS,
             "Number of experts cannot exceed %d", ES_B200_MAX_EXPERTS);
  ES_REQUIRE(num_rows >= 0, "num_rows must be non-negative");
  if (num_experts == 0 || num_rows == 0) return ES_B200_OK;
  ES_REQUIRE(input && quant_output && scale_factor && problem_sizes && expert_offsets && blockscale_offsets,
             "null pointer argument");
  ES_REQUIRE(aligned16(input) && aligned16(quant_output), "input and quant_output must be 16-byte aligned");
  ES_REQUIRE((reinterpret_cast<uintptr_t>(scale_factor) & 3u) == 0, "scale_factor must be 4-byte aligned");

  const bool wide = (reinterpret_cast<uintptr_t>(input) & 31u) == 0;      // 256-bit loads
  const bool bf16 = input_dtype == ES_B200_BF16;
  auto launch = bf16 ? (wide ? launch_quant<__nv_bfloat16, kSiluMul, true> : launch_quant<__nv_bfloat16, kSiluMul, false>)
                     : (wide ? launch_quant<__half, kSiluMul, true> : launch_quant<__half, kSiluMul, false>);
  return launch(input, problem_sizes, expert_offsets, blockscale_offsets, quant_output, scale_factor, num_experts,
                num_rows, k, static_cast<cudaStream_t>(stream));
}
}  // namespace es_b200

extern "C" int es_b200_mxfp8_grouped_quant(const void* input, int input_dtype, const int32_t* problem_sizes,
                                           const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                           void* quant_output, uint8_t* scale_factor, int num_experts,
                                           int64_t num_rows, int k, void* stream) {
  es_b200::NvtxRange nvtx_range("es_b200_mxfp8_grouped_quant");
  return es_b200::quant_impl<false>(input, input_dtype, problem_sizes, expert_offsets, blockscale_offsets, quant_output,
                                    scale_factor, num_experts, num_rows, k, stream);
}

extern "C" int es_b200_mxfp8_silu_mul_grouped_quant(const void* gate_up, int input_dtype, const int32_t* problem_sizes,
                                                    const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                                    void* quant_output, uint8_t* scale_factor, int num_experts,
                                                    int64_t num_rows, int k, void* stream) {
  es_b200::NvtxRange nvtx_range("es_b200_mxfp8_silu_mul_grouped_quant");
  return es_b200::quant_impl<true>(gate_up, input_dtype, problem_sizes, expert_offsets, blockscale_offsets, quant_output,
                                   scale_factor, num_experts, num_rows, k, stream);
}
