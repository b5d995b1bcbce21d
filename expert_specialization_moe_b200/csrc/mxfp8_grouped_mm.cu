// MXFP8 block-scaled grouped GEMM for sm_100a: the C entries, their checks, and what one launch is given.  The kernel is in
// mxfp8_grouped_mm_pair.cu.
//
// Per expert e:  d[off_e + i, n] = sum_k a[off_e + i, k] * 2^(sfa-127) * b[e, n, k] * 2^(sfb-127), fp32 accumulate.
#include "common.cuh"
#include "epilogue.cuh"
#include "grouped_mm_call.cuh"
#include "work_items.cuh"

namespace es_b200 {

namespace ep {    // expert-parallel dispatch / combine kernels (ep_dispatch_combine.cu)
int read_and_clear_status(uint32_t* out);
}
namespace route {  // expert-parallel routing tables (ep_route.cu)
int read_and_clear_status(uint32_t* out);
}
namespace bw {    // FP8-blockwise kernel (fp8_blockwise_grouped_mm.cu)
int read_and_clear_status(uint32_t* out);
}
}  // namespace es_b200

extern "C" size_t es_b200_grouped_mm_scratch_bytes(int, int64_t, int, int) {
  return es_b200::GROUPED_MM_SCRATCH_BYTES;
}

namespace es_b200 {
static int grouped_mm_impl(const void* a, const void* b, const uint8_t* sfa, const uint8_t* sfb, void* d, int out_dtype,
                           const int32_t* problem_sizes, const int32_t* expert_offsets,
                           const int32_t* blockscale_offsets, int num_experts, int64_t num_rows, int n, int k,
                           int64_t sfa_rows, const RowScatter& scatter, uint8_t* scales_out, void* scratch,
                           size_t scratch_bytes, void* stream) {
  // scales_out: silu(gate) * up requantised into d (codes) and scales_out; n is then the number of gate rows
  ES_REQUIRE(out_dtype == ES_B200_BF16 || out_dtype == ES_B200_FP16, "dtype must be kFloat16 or kBFloat16");
  ES_REQUIRE(k > 0 && k % 128 == 0, "k should align 128");
  ES_REQUIRE(n > 0 && n % 128 == 0, "n should align 128");
  ES_REQUIRE(num_experts >= 0 && num_experts <= ES_B200_MAX_EXPERTS, "Number of experts cannot exceed %d",
             ES_B200_MAX_EXPERTS);
  ES_REQUIRE(num_rows >= 0 && num_rows < (int64_t)1 << 31, "num_rows out of range");
  ES_REQUIRE((int64_t)num_experts * n * (scales_out ? 2 : 1) < (int64_t)1 << 31, "num_experts * n out of range");
  if (num_experts == 0 || num_rows == 0) return ES_B200_OK;
  ES_REQUIRE(a && b && sfa && sfb && (d || scatter.meta) && problem_sizes && expert_offsets && blockscale_offsets,
             "null pointer argument");
  ES_REQUIRE(aligned16(a) && aligned16(b) && aligned16(sfa) && aligned16(sfb), "a, b, sfa, sfb must be 16-byte aligned");
  ES_REQUIRE(aligned16(d), "d must be 16-byte aligned");
  ES_REQUIRE(sfa_rows >= 0, "sfa_rows must be non-negative");
  if (scratch != nullptr) {
    if (scratch_bytes < GROUPED_MM_SCRATCH_BYTES)
      return fail(ES_B200_ERR_SCRATCH_TOO_SMALL, "scratch holds %zu bytes, es_b200_grouped_mm_scratch_bytes asks for %zu",
                  scratch_bytes, GROUPED_MM_SCRATCH_BYTES);
    ES_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 15u) == 0, "scratch must be 16-byte aligned");
  }
  // One launch per call, whatever the row counts are: problem sizes live on the device, the work list is made there.
  const Tunables& tn = tunables();
  mm::CallArgs c = {};
  c.a = a;
  c.b = b;
  c.sfa = sfa;
  c.sfb = sfb;
  c.d = d;
  c.scales = scales_out;
  c.ps = problem_sizes;
  c.eo = expert_offsets;
  c.bo = blockscale_offsets;
  c.num_experts = num_experts;
  c.num_rows = num_rows;
  c.n = n;
  c.k = k;
  c.sfa_rows = sfa_rows;
  c.scatter = &scatter;
  c.heavy_min = tn.mm_heavy_min_rows > 0 ? tn.mm_heavy_min_rows : kHeavyMinRows;
  c.max_pairs = tn.mm_pair_max_clusters;
  c.counters = (tn.mm_dynamic && scratch) ? static_cast<uint32_t*>(scratch) : nullptr;
  // the kernel's prologue may run while the stream's earlier work drains (it waits for that work before it reads anything)
  c.overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  c.overlap.val.programmaticStreamSerializationAllowed = 1;
  c.stream = static_cast<cudaStream_t>(stream);
  if (scales_out != nullptr) return mm::launch_silu_mul_quant(c);
  return out_dtype == ES_B200_BF16 ? mm::launch_bf16(c) : mm::launch_fp16(c);
}
}  // namespace es_b200

extern "C" int es_b200_mxfp8_grouped_mm(const void* a, const void* b, const uint8_t* sfa, const uint8_t* sfb, void* d,
                                        int out_dtype, const int32_t* problem_sizes, const int32_t* expert_offsets,
                                        const int32_t* blockscale_offsets, int num_experts, int64_t num_rows, int n,
                                        int k, int64_t sfa_rows, void* scratch, size_t scratch_bytes, void* stream) {
  es_b200::NvtxRange nvtx_range("es_b200_mxfp8_grouped_mm");
  es_b200::RowScatter dense = {};
  return es_b200::grouped_mm_impl(a, b, sfa, sfb, d, out_dtype, problem_sizes, expert_offsets, blockscale_offsets,
                                  num_experts, num_rows, n, k, sfa_rows, dense, nullptr, scratch, scratch_bytes, stream);
}

extern "C" int es_b200_mxfp8_grouped_mm_silu_mul_quant(const void* a, const void* b, const uint8_t* sfa, const uint8_t* sfb,
                                                       void* quant_output, uint8_t* scale_factor,
                                                       const int32_t* problem_sizes, const int32_t* expert_offsets,
                                                       const int32_t* blockscale_offsets, int num_experts,
                                                       int64_t num_rows, int inter, int k, int64_t sfa_rows, void* scratch,
                                                       size_t scratch_bytes, void* stream) {
  es_b200::NvtxRange nvtx_range("es_b200_mxfp8_grouped_mm_silu_mul_quant");
  using namespace es_b200;
  RowScatter dense = {};
  ES_REQUIRE(num_experts == 0 || num_rows == 0 || scale_factor != nullptr, "null pointer argument");
  return grouped_mm_impl(a, b, sfa, sfb, quant_output, ES_B200_BF16, problem_sizes, expert_offsets, blockscale_offsets,
                         num_experts, num_rows, inter, k, sfa_rows, dense, scale_factor, scratch, scratch_bytes, stream);
}

extern "C" int es_b200_mxfp8_grouped_mm_scatter(const void* a, const void* b, const uint8_t* sfa, const uint8_t* sfb,
                                                int out_dtype, const int32_t* problem_sizes,
                                                const int32_t* expert_offsets, const int32_t* blockscale_offsets,
                                                int num_experts, int64_t num_rows, int n, int k, int64_t sfa_rows,
                                                const int32_t* row_meta, const void* const* peer_out, int world,
                                                int64_t slots_per_gpu, void* scratch, size_t scratch_bytes,
                                                void* stream) {
  es_b200::NvtxRange nvtx_range("es_b200_mxfp8_grouped_mm_scatter");
  using namespace es_b200;
  ES_REQUIRE(world >= 1 && world <= SCATTER_MAX_GPUS, "world size must be in [1, %d]", SCATTER_MAX_GPUS);
  ES_REQUIRE(row_meta && peer_out, "null pointer argument");
  ES_REQUIRE((reinterpret_cast<uintptr_t>(row_meta) & 7u) == 0, "row_meta must be 8-byte aligned");
  ES_REQUIRE(slots_per_gpu >= 0, "slots_per_gpu out of range");
  RowScatter sc = {};
  sc.meta = reinterpret_cast<const int2*>(row_meta);
  sc.gpus = world;
  sc.slots = slots_per_gpu;
  for (int i = 0; i < world; ++i) {
    ES_REQUIRE(peer_out[i] != nullptr && aligned16(peer_out[i]), "peer output %d must be a 16-byte aligned pointer", i);
    sc.base[i] = const_cast<void*>(peer_out[i]);
  }
  return grouped_mm_impl(a, b, sfa, sfb, nullptr, out_dtype, problem_sizes, expert_offsets, blockscale_offsets,
                         num_experts, num_rows, n, k, sfa_rows, sc, nullptr, scratch, scratch_bytes, stream);
}

extern "C" int es_b200_check_status(void* stream, uint32_t* raw_status) {
  using namespace es_b200;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  ES_CUDA_TRY(cudaStreamSynchronize(s));
  uint32_t v = 0, v2 = 0;
  int rc2 = mm::read_and_clear_status(&v);
  if (rc2 != ES_B200_OK) return rc2;
  rc2 = bw::read_and_clear_status(&v2);
  if (rc2 != ES_B200_OK) return rc2;
  v |= v2;
  rc2 = ep::read_and_clear_status(&v2);
  if (rc2 != ES_B200_OK) return rc2;
  v |= v2;
  rc2 = route::read_and_clear_status(&v2);
  if (rc2 != ES_B200_OK) return rc2;
  v |= v2;
  if (raw_status) *raw_status = v;
  if (v != 0) note_device_error();
  if (v != 0)
    return fail(ES_B200_ERR_DEVICE_TIMEOUT,
                "a bounded device-side wait gave up or an index was out of range (status bits 0x%x)", v);
  return ES_B200_OK;
}
