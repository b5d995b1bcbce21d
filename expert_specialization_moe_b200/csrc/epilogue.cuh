// Accumulator -> global memory: conversions, wide stores, and the scattered destination of output rows.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sm100_ptx.cuh"

namespace es_b200 {

// Optional destination map of the output rows (expert-parallel combine fused into the GEMM): output row r goes to row
// meta[r].y of the [slots, n] array base[meta[r].x] — another GPU's buffer mapped into this process, or a local one —
// instead of row r of d.  meta == nullptr: dense output.  Entries out of range are skipped and reported.
constexpr int SCATTER_MAX_GPUS = 16;
constexpr uint32_t ERR_SCATTER_DESTINATION = 0x40000u;
struct RowScatter {
  const int2* meta;
  void* base[SCATTER_MAX_GPUS];
  long long slots;
  int gpus;
};

template <typename OutT>
__device__ __forceinline__ OutT out_from_f32(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 out_from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half out_from_f32<__half>(float v) { return __float2half_rn(v); }

// Scatter destination of output row `row` as a pointer to the warp's first column in that row, or null (entry out of
// range: reported; row past the valid ones: silent).
template <typename OutT>
__device__ __forceinline__ OutT* scatter_row_ptr(const RowScatter& scatter, int64_t row, bool in_range, int64_t ld,
                                                 int col_off, uint32_t* status) {
  if (!in_range) return nullptr;
  const int2 m = scatter.meta[row];
  if (m.x >= 0 && m.x < scatter.gpus && m.y >= 0 && m.y < scatter.slots)
    return static_cast<OutT*>(scatter.base[m.x]) + (int64_t)m.y * ld + col_off;
  atomicOr(status, ERR_SCATTER_DESTINATION);
  return nullptr;
}

template <typename OutT>
__device__ __forceinline__ uint32_t pack_pair_from_f32(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack_pair_from_f32<__nv_bfloat16>(float lo, float hi) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}
template <>
__device__ __forceinline__ uint32_t pack_pair_from_f32<__half>(float lo, float hi) {
  const __half2 p = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&p);
}

// 32 bytes per thread to global memory: one 256-bit store where the address allows it, two 128-bit stores otherwise
// (out is at least 16-byte aligned)
__device__ __forceinline__ void store_32B(void* out, const uint32_t (&w)[8], bool aligned32) {
  if (aligned32) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(out), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    static_cast<uint4*>(out)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    static_cast<uint4*>(out)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

}  // namespace es_b200
