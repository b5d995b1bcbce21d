// What the entries of the MXFP8 grouped GEMM (mxfp8_grouped_mm.cu) hand to its kernel's launch (mxfp8_grouped_mm_pair.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "epilogue.cuh"

namespace es_b200 {
namespace mm {

struct CallArgs {
  const void* a;
  const void* b;
  const uint8_t* sfa;
  const uint8_t* sfb;
  void* d;                 // silu_mul_quant: the codes
  uint8_t* scales;         // silu_mul_quant: their scale bytes
  const int32_t* ps;
  const int32_t* eo;
  const int32_t* bo;
  int num_experts;
  int64_t num_rows;
  int n, k;
  int64_t sfa_rows;
  const RowScatter* scatter;
  int heavy_min;           // experts with at least this many rows come first in the work list
  int max_pairs;           // cap of the grid in CTA pairs (0 = as many as fit on the device)
  uint32_t* counters;      // work counters in the caller's scratch; null: items are dealt round-robin over the grid
  cudaLaunchAttribute overlap;
  cudaStream_t stream;
};

int launch_bf16(const CallArgs& c);
int launch_fp16(const CallArgs& c);
int launch_silu_mul_quant(const CallArgs& c);   // n: gate rows per expert
int read_and_clear_status(uint32_t* out);

}  // namespace mm
}  // namespace es_b200
