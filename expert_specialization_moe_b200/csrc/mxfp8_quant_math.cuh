// MXFP8 quantisation arithmetic shared by the grouped quant kernel and the expert-parallel dispatch kernel.
//
// Arithmetic contract (bit-exact with the reference kernel, es_sm100_mxfp8_blockscaled_group_quant.cuh:36-134):
//   amax  = max |x_i| over the 32-block, NaN members dropped (max.bf16x2 / max.f16x2 semantics)
//   s     = fp32(amax) * rcp.approx.ftz.f32(448.0f)
//   sf    = cvt.rp.satfinite.ue8m0x2.f32(s)
//   inv   = amax != 0 ? rcp.approx.ftz.f32(float(sf)) : 0
//   code  = cvt.rn.satfinite.e4m3x2.f32(fp32(x_i) * inv)
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

namespace es_b200 {

__device__ __forceinline__ float rcp_approx_ftz(float a) {
  float b;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(a));   // pure: may be hoisted / scheduled freely
  return b;
}

// (ld.global.nc: for kernels that start after the producer of the memory has finished, not for those launched with
// programmatic stream serialisation, during whose life it may still be written)
__device__ __forceinline__ uint4 ld_stream_16B(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// Predicated streaming accesses: no branch around them, and the registers of a load that is off keep their value.
// 32 bytes per lane in one instruction (sm_100); p must be 32-byte aligned
__device__ __forceinline__ void ld_stream_32B_if(const void* p, bool on, uint32_t (&v)[8]) {
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "setp.ne.b32 P, %9, 0;\n\t"
      "@P ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
      "}"
      : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
      : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ld_stream_16B_if(const void* p, bool on, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "setp.ne.b32 P, %5, 0;\n\t"
      "@P ld.global.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];\n\t"
      "}"
      : "+r"(a), "+r"(b), "+r"(c), "+r"(d)
      : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void st_stream_16B_if(void* p, bool on, const uint4& v) {
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "setp.ne.b32 P, %5, 0;\n\t"
      "@P st.global.cs.v4.b32 [%0], {%1,%2,%3,%4};\n\t"
      "}" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"((int)on)
      : "memory");
}
__device__ __forceinline__ void st_4B_if(void* p, bool on, uint32_t v) {
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "setp.ne.b32 P, %2, 0;\n\t"
      "@P st.global.b32 [%0], %1;\n\t"
      "}" ::"l"(p), "r"(v), "r"((int)on)
      : "memory");
}

__device__ __forceinline__ float ex2_approx_ftz(float a) {
  float b;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(a));
  return b;
}

// two fp32 operations per instruction (sm_100), each rounded to nearest as the scalar form
__device__ __forceinline__ unsigned long long pack_f32x2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 unpack_f32x2(unsigned long long a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack_f32x2(a)), "l"(pack_f32x2(b)));
  return unpack_f32x2(r);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack_f32x2(a)), "l"(pack_f32x2(b)));
  return unpack_f32x2(r);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack_f32x2(a)), "l"(pack_f32x2(b)), "l"(pack_f32x2(c)));
  return unpack_f32x2(r);
}

template <typename T>
struct Vec2;
template <>
struct Vec2<__nv_bfloat16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ float2 to_float2(type v) { return __bfloat1622float2(v); }
  static __device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ float from_bits(uint32_t v) { return __uint_as_float(v << 16); }
  static __device__ __forceinline__ type from_floats(float a, float b) { return __floats2bfloat162_rn(a, b); }
};
template <>
struct Vec2<__half> {
  using type = __half2;
  static __device__ __forceinline__ float2 to_float2(type v) { return __half22float2(v); }
  static __device__ __forceinline__ float to_float(__half v) { return __half2float(v); }
  static __device__ __forceinline__ float from_bits(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }
  static __device__ __forceinline__ type from_floats(float a, float b) { return __floats2half2_rn(a, b); }
};

// Quantise the 8 elements this lane holds; the four lanes of a quad share one 32-element block.
// Returns the block's UE8M0 byte (same value in all four lanes); writes the 8 codes to `codes`.
template <typename T>
__device__ __forceinline__ uint32_t quantize8(const uint4& raw, uint2& codes) {
  using V2 = typename Vec2<T>::type;
  V2 v[4];
  v[0] = *reinterpret_cast<const V2*>(&raw.x);
  v[1] = *reinterpret_cast<const V2*>(&raw.y);
  v[2] = *reinterpret_cast<const V2*>(&raw.z);
  v[3] = *reinterpret_cast<const V2*>(&raw.w);
  V2 mx = __hmax2(__hmax2(__habs2(v[0]), __habs2(v[1])), __hmax2(__habs2(v[2]), __habs2(v[3])));
  {
    uint32_t bits = *reinterpret_cast<uint32_t*>(&mx);
    uint32_t o = __shfl_xor_sync(0xffffffffu, bits, 1);
    mx = __hmax2(mx, *reinterpret_cast<V2*>(&o));
    bits = *reinterpret_cast<uint32_t*>(&mx);
    o = __shfl_xor_sync(0xffffffffu, bits, 2);
    mx = __hmax2(mx, *reinterpret_cast<V2*>(&o));
  }
  const float block_max = Vec2<T>::to_float(__hmax(mx.x, mx.y));
  float sf_val = block_max * rcp_approx_ftz(448.0f);
  __nv_fp8_e8m0 sf;
  sf.__x = __nv_cvt_float_to_e8m0(sf_val, __NV_SATFINITE, cudaRoundPosInf);
  sf_val = static_cast<float>(sf);
  const float inv = block_max != 0.f ? rcp_approx_ftz(sf_val) : 0.0f;

  uint32_t out[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float2 lo = Vec2<T>::to_float2(v[2 * i]);
    float2 hi = Vec2<T>::to_float2(v[2 * i + 1]);
    lo.x *= inv; lo.y *= inv; hi.x *= inv; hi.y *= inv;
    uint32_t p0 = __nv_cvt_float2_to_fp8x2(lo, __NV_SATFINITE, __NV_E4M3);
    uint32_t p1 = __nv_cvt_float2_to_fp8x2(hi, __NV_SATFINITE, __NV_E4M3);
    out[i] = p0 | (p1 << 16);
  }
  codes.x = out[0];
  codes.y = out[1];
  return sf.__x;
}

// max(|a|, |b|) per half, the sign of the result unspecified; NaN members dropped
template <typename T>
__device__ __forceinline__ uint32_t max_magnitude2(uint32_t a, uint32_t b);
template <>
__device__ __forceinline__ uint32_t max_magnitude2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <>
__device__ __forceinline__ uint32_t max_magnitude2<__half>(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

template <typename T>
__device__ __forceinline__ uint32_t max_magnitude16(const uint32_t (&v)[8]) {
  const uint32_t a = max_magnitude2<T>(max_magnitude2<T>(v[0], v[1]), max_magnitude2<T>(v[2], v[3]));
  const uint32_t b = max_magnitude2<T>(max_magnitude2<T>(v[4], v[5]), max_magnitude2<T>(v[6], v[7]));
  return max_magnitude2<T>(a, b);
}

// larger of the two halves, each pair compared as unsigned 16-bit numbers
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// larger magnitude of the two halves as fp32 (NaN only if both are)
template <typename T>
__device__ __forceinline__ float magnitude_of_pair(uint32_t m) {
  using V2 = typename Vec2<T>::type;
  m &= 0x7fff7fffu;
  const V2 mx = *reinterpret_cast<const V2*>(&m);
  return Vec2<T>::to_float(__hmax(mx.x, mx.y));
}

// largest |v_i| of the lane's 16 elements, NaN members dropped
template <typename T>
__device__ __forceinline__ float max_abs16(const uint32_t (&v)[8]) {
  return magnitude_of_pair<T>(max_magnitude16<T>(v));
}

// four fp32 values -> four e4m3 codes, the first in the lowest byte
__device__ __forceinline__ uint32_t e4m3x4(float2 lo, float2 hi) {
  uint32_t r;
  asm("{\n\t"
      ".reg .b16 a, b;\n\t"
      "cvt.rn.satfinite.e4m3x2.f32 a, %2, %1;\n\t"
      "cvt.rn.satfinite.e4m3x2.f32 b, %4, %3;\n\t"
      "mov.b32 %0, {a, b};\n\t"
      "}"
      : "=r"(r)
      : "f"(lo.x), "f"(lo.y), "f"(hi.x), "f"(hi.y));
  return r;
}

// Quantise the 16 elements this lane holds (largest = max_magnitude16 of them); two neighbouring lanes share one 32-element
// block.  Same arithmetic as quantize8; returns the block's UE8M0 byte in both lanes.
template <typename T>
__device__ __forceinline__ uint32_t quantize16(const uint32_t (&v)[8], uint32_t largest, uint4& codes) {
  using V2 = typename Vec2<T>::type;
  const uint32_t mx = max_magnitude2<T>(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
  const float block_max = magnitude_of_pair<T>(mx);
  const uint32_t sf = __nv_cvt_float_to_e8m0(block_max * rcp_approx_ftz(448.0f), __NV_SATFINITE, cudaRoundPosInf);
  // rcp.approx.ftz(2^(sf - 127)): 2^(127 - sf); the subnormal 2^-127 (sf = 0) counts as zero, 1 / 2^127 (254) flushes to
  // zero; a block whose 32 members are all NaN has the scale NaN (255)
  const uint32_t inv_bits = sf == 0 ? 0x7f800000u : sf == 255u ? 0x7fffffffu : (254u - sf) << 23;
  const float inv = block_max != 0.f ? __uint_as_float(inv_bits) : 0.0f;
  uint32_t out[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    out[i] = e4m3x4(mul2(Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&v[2 * i])), make_float2(inv, inv)),
                    mul2(Vec2<T>::to_float2(*reinterpret_cast<const V2*>(&v[2 * i + 1])), make_float2(inv, inv)));
  codes = make_uint4(out[0], out[1], out[2], out[3]);
  return sf;
}

// Byte offset, inside one operand's swizzled scale buffer, of the 32-bit scale word of (row r, K tile 0): 512-byte
// atoms of 128 rows x 4 K blocks, atoms K-fastest (kt = K / 128 atoms per 128 rows); the word of K tile q is q * 512
// further on.
__device__ __host__ __forceinline__ int64_t scale_word_offset(int r, int kt) {
  return (int64_t)(r >> 7) * kt * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4;
}

}  // namespace es_b200
