// What the two kernels of one FP8-blockwise grouped GEMM call share on the host.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace es_b200 {
namespace bw {

struct CallArgs {
  const void* a;
  const void* b;
  const float* sa;
  const float* sb;
  void* d;
  const int32_t* ps;
  const int32_t* eo;
  int num_experts;
  int64_t num_rows;
  int n, k;
  cudaStream_t stream;
};

constexpr int FEW_ROWS = 32;      // experts with at most this many rows: fp8_blockwise_grouped_mm.cu

// experts with more than FEW_ROWS rows (fp8_blockwise_many_rows.cu); second launch of the call
int launch_many_rows_bf16(const CallArgs& c);
int launch_many_rows_fp16(const CallArgs& c);
int read_and_clear_status_many_rows(uint32_t* out);

}  // namespace bw
}  // namespace es_b200
