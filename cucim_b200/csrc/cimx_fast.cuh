// cimx_fast.cuh — what the fast float32 kernels share: 4-wide vector types,
// exact integer widening, the narrowing casts, float32 pairs and their fused
// multiply-add, and asynchronous copies to shared memory.
#pragma once

#include "cimx_common.cuh"
#include "cimx_tma.cuh"  // smem_addr

namespace cimx {
namespace fast {

constexpr int kMaxSmem = 227 * 1024;

// ------------------------------------------------------------ vector I/O

template <class T> struct Vec4;
template <> struct Vec4<float> { using type = float4; };
template <> struct Vec4<uint16_t> { using type = ushort4; };
template <> struct Vec4<uint8_t> { using type = uchar4; };

// Exact float value of an unsigned integer below 2^23 without the conversion
// unit: the integer placed in the mantissa of 2^23, minus 2^23.
template <class T>
__device__ __forceinline__ float exact_float(T v) {
  if constexpr (sizeof(T) == 4) {
    return static_cast<float>(v);
  } else {
    return __fsub_rn(__uint_as_float(0x4B000000u | static_cast<uint32_t>(v)), 8388608.0f);
  }
}

// cast<D>(a) of an intermediate that stays on chip, as the float the next
// pass reads (out_cast writes the narrowing conversion out explicitly, so
// widening its result again keeps the narrow value)
template <class D>
__device__ __forceinline__ float narrow_float(float a) {
  if constexpr (sizeof(D) == 4) return a;
  else return exact_float(out_cast<D>(a));
}

// cast<D>(a) as stored
template <class D>
__device__ __forceinline__ D narrow_cast(float a) {
  return out_cast<D>(a);
}

template <class T> constexpr int dt_code();
template <> constexpr int dt_code<float>() { return DT_F32; }
template <> constexpr int dt_code<uint16_t>() { return DT_U16; }
template <> constexpr int dt_code<uint8_t>() { return DT_U8; }

// ------------------------------------------------------------- helpers

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <class T>
__device__ __forceinline__ void cp_async_vec4(T* dst, const T* src) {
  if constexpr (sizeof(T) == 4) cp_async16(dst, src);
  else if constexpr (sizeof(T) == 2) cp_async8(dst, src);
  else cp_async4(dst, src);
}


// Two float32 lanes in one 64-bit register (x in the low half).
using f2 = unsigned long long;

__device__ __forceinline__ f2 pack2(float x, float y) {
  return (static_cast<f2>(__float_as_uint(y)) << 32) | __float_as_uint(x);
}
__device__ __forceinline__ float lo2(f2 v) { return __uint_as_float(static_cast<unsigned>(v)); }
__device__ __forceinline__ float hi2(f2 v) {
  return __uint_as_float(static_cast<unsigned>(v >> 32));
}

// d = fma(a, b, c) on both lanes, each an IEEE float32 FMA rounded to nearest
// (bit-identical to fmaf on each lane).
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

}  // namespace fast
}  // namespace cimx
