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
// Eight lanes take a tile, sixteen elements each, a CTA 32 consecutive tiles per step.  The steps of all experts form one
// flat list (a per-CTA prefix scan over the row counts) that the resident CTAs share evenly: neither the split of the rows
// between experts nor k leaves lanes or CTAs idle.  Zeroing the scale bytes of the padding rows is steps of its own, in
// 16-byte pieces: in a decode call they are as many bytes as the codes.
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
constexpr int QUANT_WARP_TILES = 4;           // a warp's four groups of eight lanes, one 128-element K tile each
constexpr int QUANT_STEP_TILES = QUANT_WARPS * QUANT_WARP_TILES;
constexpr int QUANT_PAD_ATOMS = 16;           // scale atoms per warp and step of padding work
// Consecutive steps that a CTA takes before it moves on by a grid's worth: its equal share of the list in one stretch, or
// eight where the share is long and the kernel is bound by memory: 592 streams far apart cost bandwidth, the uneven last
// round of chunks costs the most where there are few rounds.  One stretch / chunks of 8, us: share 16 23.6 / 26.7, 20
// 28.3 / 30.0, 24 33.5 / 34.3, 26 36.1 / 36.8, 28 38.6 / 38.2, 30 41.2 / 38.7, 36 48.9 / 46.7, 48 65.5 / 60.5 (k = 768;
// k = 2048 and 7168 cross between 22 and 28 too); 97 (32768 x 7168) 128 / 125.  Chunks of 4 and 2 are slower than of 8
// there.  With silu, bound by its arithmetic, no difference (131072 x 768), and the last round is not paid for.
constexpr int QUANT_CHUNK = 8, QUANT_LONG_SHARE = 27;
// registers: two steps of input in flight per warp; the fused variant holds gate and up of both
constexpr int QUANT_MIN_BLOCKS = 4, QUANT_MIN_BLOCKS_SILU = 3;

// exact arithmetic of an unfused silu(gate.float()) * up.float() -> T: accurate expf, IEEE division and multiply
__device__ __forceinline__ float silu_mul_exact(float g, float u) { return (g / (1.0f + expf(-g))) * u; }

// act = round_to_T( silu(gate) * up ) on 16 elements; the codes and scale of their block are bit for bit those of
// silu_mul_exact's values, for a third of its instructions.  p = g * rcp(1 + 2^(-g log2 e)) * u with the hardware
// approximations is within `eps` (relative) of the exact sequence's fp32 value, so wherever p (1 - eps) and p (1 + eps)
// round to the same 16-bit value, that value is the answer (rounding is monotonic); the few pairs where they do not (of
// N(0, 1) values 0.05 % of the elements in bf16, 0.4 % in fp16) take the exact sequence.
// Error of p against the exact sequence, in units of 2^-24: 2^x 4 (2 ulp), its argument 1.22 |g| (the product g log2 e and
// the constant; at most 0.45 for g > 0, where 2^x is at most e^-g of the sum), reciprocal 2 (1 ulp), sum and two products
// 3 x 1; exact sequence: expf 2 (1 ulp), sum, quotient and product 3 x 1; the factors 1 +- eps and their products 2.
// 16 + 1.22 |g| in all; eps = (20 + 1.25 |g|) 2^-24 with the lane's lowest g.  (|g| < 2^-124 makes g / 2 subnormal: at
// most 5 more, and only where it is large enough for an error to round away from it.)
// The bound does not hold for g < -64 (1 + 2^x may leave the range of the reciprocal, p is then accurate or a zero of the
// right sign) and for |p| near the fp32 subnormals.  Both are values that the block's scale turns into a signed zero,
// whatever their digits, unless all the lane's values are that small: |p| <= 2^-86 |u| for the former, so a largest value
// above 2^20 times these limits settles it (scaled to 448, they are below 2^-11, half of the smallest code is 2^-10).  Lanes
// that it does not settle — none in practice but those whose values are all zero — take the exact sequence for every
// element that is not a zero by its factors.  (Whole lanes by the exact sequence because of one zero or one large gate cost
// a warp's step eight serial turns: 131072 x 768 bf16 with 1 % of zeros 312 us, 96 this way; 50-fold outliers 226, 99.)
// fp16 products are zero or at least 2^-110.
// `largest`: magnitudes of the lane's largest values, as max_magnitude16 gives them.
template <typename T>
__device__ __forceinline__ void silu_mul16(const uint32_t (&g)[8], const uint32_t (&u)[8], uint32_t (&out)[8],
                                           uint32_t& largest) {
  using V2 = typename Vec2<T>::type;
  const uint32_t low2 = max_u16x2(max_u16x2(max_u16x2(g[0], g[1]), max_u16x2(g[2], g[3])),
                                  max_u16x2(max_u16x2(g[4], g[5]), max_u16x2(g[6], g[7])));
  const float low = Vec2<T>::from_bits(max(low2 >> 16, low2 & 0xffffu));   // negative values sort highest, most negative last
  const bool in_range = low >= -64.0f;                                     // no: a lower one or a NaN among them
  const float eps = fmaf(in_range ? fmaxf(-low, 0.0f) : 64.0f, 7.450580597e-8f, 1.192092896e-6f);   // (20 + 1.25 |g|) 2^-24
  const float2 up = make_float2(1.0f + eps, 1.0f + eps), down = make_float2(1.0f - eps, 1.0f - eps);
  uint32_t undecided = 0u;      // one bit per pair
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 gf = Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&g[i]));
    const float2 uf = Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&u[i]));
    const float2 t = mul2(gf, make_float2(-1.4426950408889634f, -1.4426950408889634f));
    const float2 d = add2(make_float2(ex2_approx_ftz(t.x), ex2_approx_ftz(t.y)), make_float2(1.0f, 1.0f));
    const float2 p = mul2(mul2(gf, make_float2(rcp_approx_ftz(d.x), rcp_approx_ftz(d.y))), uf);
    const float2 hi = mul2(p, up), lo = mul2(p, down);      // a zero keeps its sign in both
    const V2 r_hi = Vec2<T>::from_floats(hi.x, hi.y), r_lo = Vec2<T>::from_floats(lo.x, lo.y);
    out[i] = *reinterpret_cast<const uint32_t*>(&r_hi);
    if (out[i] != *reinterpret_cast<const uint32_t*>(&r_lo)) undecided |= 1u << i;
  }
  largest = max_magnitude16<T>(out);
  float limit = std::is_same<T, __nv_bfloat16>::value ? 8.271806125530277e-25f : -1.0f;      // 2^-80
  if (!in_range) limit = fmaxf(limit, max_abs16<T>(u) * 1.3552527156068805e-20f);            // 2^-66 |u|
  if (!(magnitude_of_pair<T>(largest) > limit)) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t gm = g[i] & 0x7fff7fffu, um = u[i] & 0x7fff7fffu;
      if (((gm & 0xffffu) != 0u && (um & 0xffffu) != 0u) || (gm >> 16 != 0u && um >> 16 != 0u)) undecided |= 1u << i;
    }
  }
  if (undecided == 0u) return;
  // no branch above: the sixteen chains overlap.  One undecided pair per turn here (bf16: a turn in 21 % of a warp's steps;
  // fp16: 0.9 turns per step).
  do {
    const int i = __ffs((int)undecided) - 1;
    undecided &= undecided - 1;
    uint32_t gw = g[0], uw = u[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) {
      if (i == j) { gw = g[j]; uw = u[j]; }
    }
    const float2 gf = Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&gw));
    const float2 uf = Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&uw));
    const V2 r = Vec2<T>::from_floats(silu_mul_exact(gf.x, uf.x), silu_mul_exact(gf.y, uf.y));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (i == j) out[j] = *reinterpret_cast<const uint32_t*>(&r);
    }
  } while (undecided != 0u);
  largest = max_magnitude16<T>(out);
}

// 32 bytes of input per lane (v is left alone where `on` is false): one 256-bit load where the tensor starts on a 32-byte
// boundary (tiles are multiples of 256 bytes), two 128-bit loads otherwise
template <bool kWide>
__device__ __forceinline__ void load_16_elements(const void* p, bool on, uint32_t (&v)[8]) {
  if constexpr (kWide) {
    ld_stream_32B_if(p, on, v);
  } else {
    ld_stream_16B_if(p, on, v[0], v[1], v[2], v[3]);
    ld_stream_16B_if(static_cast<const uint8_t*>(p) + 16, on, v[4], v[5], v[6], v[7]);
  }
}

// kSiluMul = false: input [rows, k].  kSiluMul = true: input [rows, 2k] = gate | up, quantises silu(gate) * up.
// The inputs are not __restrict__: the kernel may start while their producer still runs (programmatic launch), and the
// read-only path wants memory that nothing writes during the kernel's life.
template <typename T, bool kSiluMul, bool kWide>
__global__ void __launch_bounds__(QUANT_THREADS, kSiluMul ? QUANT_MIN_BLOCKS_SILU : QUANT_MIN_BLOCKS)
mxfp8_group_quant_kernel(const T* input, const int* problem_sizes, const int* expert_offsets, const int* blockscale_offsets,
                         uint8_t* __restrict__ quant_output, uint8_t* __restrict__ scale_factor, int num_experts,
                         int k) {
  __shared__ int table[ES_B200_MAX_EXPERTS + 1];
  __shared__ int warp_sums[32];

  const int kt = k >> 7;                          // K tiles (= 32-bit scale words) per row
  const int step_rows = QUANT_STEP_TILES / kt, step_q = QUANT_STEP_TILES - step_rows * kt;
  const int pad_steps = (kt + QUANT_WARPS * QUANT_PAD_ATOMS - 1) / (QUANT_WARPS * QUANT_PAD_ATOMS);
  // (a tile is at least 256 bytes of input: 32 bits count the tiles of any tensor that fits the GPU)
  auto data_steps = [&](int m) { return (int)(((uint32_t)m * (uint32_t)kt + QUANT_STEP_TILES - 1u) / QUANT_STEP_TILES); };
  pdl_wait_prior_grid();
  block_exclusive_scan(num_experts, table, warp_sums, [&](int e) {
    const int m = problem_sizes[e * 3];
    return m > 0 ? data_steps(m) + ((m & 127) ? pad_steps : 0) : 0;
  });
  const ExpertTable tab = fill_expert_table(table, num_experts, problem_sizes, expert_offsets, blockscale_offsets);
  __syncthreads();
  pdl_launch_dependents();
  const int total = tab.prefix[num_experts];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first_tile = warp * QUANT_WARP_TILES;                // of a step's 32 tiles
  const int group = lane >> 3, l8 = lane & 7;     // this lane's tile of the warp's four, and its 16 elements of the tile

  const int share = (total + (int)gridDim.x - 1) / (int)gridDim.x;
  const int chunk = (kSiluMul || share <= QUANT_LONG_SHARE) ? share : QUANT_CHUNK;
  int u = (int)blockIdx.x * chunk, end = min(u + chunk, total);
  if (u >= total) return;
  int e = upper_bound_expert(tab.prefix, num_experts, u);
  for (int run; u < end; ) {
    while (tab.prefix[e + 1] <= u) ++e;             // empty experts share their prefix with the next one
    const int i = u - tab.prefix[e];
    const int m = tab.m(e);
    uint8_t* sf_expert = scale_factor + (int64_t)tab.scale0(e) * (k >> 5);
    const int n_data = data_steps(m);
    if (i >= n_data) {
      run = 1;
      // scale bytes of the padding rows m .. align128(m) - 1: lane j clears, in each atom, the words of its line (rows
      // j, j + 32, j + 64, j + 96 of the last 128) that belong to rows past the end
      const int last = m & 127;
      const int first_word = last <= lane ? 0 : (last - lane + 31) >> 5;      // 0 .. 4
      uint8_t* line = sf_expert + (int64_t)(m >> 7) * kt * 512 + lane * 16;
      // (atoms dealt to the warps one by one: in runs of sixteen, k <= 2048 left seven of the eight without any, 4.6 us
      // against 2.9 for 16 rows x 2048)
      const int q0 = (i - n_data) * QUANT_WARPS * QUANT_PAD_ATOMS;
      for (int q = q0 + warp; q < min(kt, q0 + QUANT_WARPS * QUANT_PAD_ATOMS); q += QUANT_WARPS) {
        uint32_t* words = reinterpret_cast<uint32_t*>(line + (int64_t)q * 512);
        if (first_word == 0 && (reinterpret_cast<uintptr_t>(words) & 15u) == 0) {
          *reinterpret_cast<uint4*>(words) = make_uint4(0, 0, 0, 0);
        } else {
          for (int w = first_word; w < 4; ++w) words[w] = 0u;
        }
      }
    } else {
      run = min(end - u, n_data - i);
      const uint32_t t0 = (uint32_t)i * QUANT_STEP_TILES + (uint32_t)(first_tile + group);    // this lane group's first tile
      // tiles from the warp's first on; the same number of steps for all its lanes: the shuffles need them
      const int warp_left = (int)((uint32_t)m * (uint32_t)kt - (uint32_t)i * QUANT_STEP_TILES) - first_tile;
      const int n_steps = min(run, (warp_left + QUANT_STEP_TILES - 1) / QUANT_STEP_TILES);
      int row = (int)(t0 / (uint32_t)kt);
      int q = (int)(t0 - (uint32_t)row * (uint32_t)kt);
      int load_q = q;
      const int64_t row0 = tab.row0(e);
      // gate tiles of one row and the next are kt tiles further apart than those inside a row
      const T* src = input + (kSiluMul ? row0 * 2 * kt + t0 + (int64_t)row * kt : row0 * kt + t0) * 128 + l8 * 16;
      uint8_t* dst = quant_output + (row0 * kt + t0) * 128 + l8 * 16;
      int left = warp_left - group;                            // tiles from this lane group's next one on: to store,
      int load_left = min(left, n_steps * QUANT_STEP_TILES);   // to load (of this run only: the next one loads its own)

      auto load = [&](uint32_t (&g)[8], uint32_t (&up)[8]) {
        const bool on = load_left > 0;
        load_left -= QUANT_STEP_TILES;
        load_16_elements<kWide>(src, on, g);
        if constexpr (kSiluMul) {
          load_16_elements<kWide>(src + k, on, up);
          load_q += step_q;
          int skip = step_rows;
          if (load_q >= kt) { load_q -= kt; ++skip; }
          src += (QUANT_STEP_TILES + skip * kt) * 128;
        } else {
          src += QUANT_STEP_TILES * 128;
        }
      };
      // quantises the step in (g, up); the loads of the step after next go out in front of the quantisation, into `next`
      // (silu: into the registers that the activation has just freed)
      auto step = [&](uint32_t (&g)[8], uint32_t (&up)[8], uint32_t (&next)[8]) {
        uint4 codes;
        uint32_t sf;
        if constexpr (kSiluMul) {
          uint32_t v[8], largest;
          silu_mul16<T>(g, up, v, largest);
          load(g, up);
          sf = quantize16<T>(v, largest, codes);
        } else {
          load(next, up);
          sf = quantize16<T>(g, max_magnitude16<T>(g), codes);
        }
        // the four scale bytes of the tile as one aligned 32-bit word (two lanes hold the byte of a 32-element block)
        uint32_t w = sf << ((l8 >> 1) * 8);
        w |= __shfl_xor_sync(0xffffffffu, w, 2);
        w |= __shfl_xor_sync(0xffffffffu, w, 4);
        const bool on = left > 0;
        left -= QUANT_STEP_TILES;
        st_stream_16B_if(dst, on, codes);
        dst += QUANT_STEP_TILES * 128;
        // (an expert's scale bytes are 1/64 of its input: 32 bits address them)
        const uint32_t at = ((uint32_t)(row >> 7) * (uint32_t)kt + (uint32_t)q) * 512u + (row & 31) * 16 + ((row & 127) >> 5) * 4;
        st_4B_if(sf_expert + at, on && l8 == 0, w);
        row += step_rows;
        q += step_q;
        if (q >= kt) { q -= kt; ++row; }
      };
      // two steps in flight besides the one at work; tiles past the end quantise zeros and store nothing
      constexpr int BUFFERS = kSiluMul ? 2 : 3;
      uint32_t raw[BUFFERS][8], raw_up[2][8];
#pragma unroll
      for (int b = 0; b < BUFFERS; ++b) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          raw[b][j] = 0u;
          if (b < 2) raw_up[b][j] = 0u;
        }
      }
      load(raw[0], raw_up[0]);
      load(raw[1], raw_up[1]);
      for (int s = 0; s < n_steps; ++s) {
        step(raw[0], raw_up[0], raw[BUFFERS - 1]);
        if (++s == n_steps) break;
        step(raw[1], raw_up[1], raw[0]);
        if constexpr (BUFFERS == 3) {
          if (++s == n_steps) break;
          step(raw[2], raw_up[0], raw[1]);
        }
      }
    }
    u += run;
    if (u >= end) {                                 // on to the CTA's next chunk
      u += ((int)gridDim.x - 1) * chunk;
      end = min(u + chunk, total);
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
  // at most one partial step and the padding steps per expert on top of the full steps of num_rows rows
  const int kt = k >> 7;
  const int64_t max_ctas = (num_rows * kt + QUANT_STEP_TILES - 1) / QUANT_STEP_TILES +
                           (int64_t)num_experts * (1 + (kt + QUANT_WARPS * QUANT_PAD_ATOMS - 1) / (QUANT_WARPS * QUANT_PAD_ATOMS));
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
                                 blockscale_offsets, static_cast<uint8_t*>(quant_output), scale_factor, num_experts, k));
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
