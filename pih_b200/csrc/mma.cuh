// Warp-level tensor-core helpers (mma.sync m16n8k16 on bf16, ldmatrix, cp.async) for kernels whose tiles are too
// small or too irregular for tcgen05.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace pih {
namespace mma {

__device__ __forceinline__ void copy_async_16(void* smem, const void* gmem) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
// (zeros where there is nothing; ``gmem`` is a readable address all the same)
__device__ __forceinline__ void copy_async_16_or_zero(void* smem, const void* gmem, bool there) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(there ? 16 : 0));
}
__device__ __forceinline__ void copy_async_4(void* smem, const void* gmem) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void load_matrices(uint32_t (&r)[4], const void* smem) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void load_matrices_transposed(uint32_t (&r)[4], const void* smem) {
  const uint32_t s = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
// c += a (16 x 16, row-major) . b (16 x 8, column-major), 32-bit accumulation
__device__ __forceinline__ void multiply_add(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// the part of (lo, hi) that their bf16 roundings ``packed`` (= pack(lo, hi)) leave out, as bf16: a bf16 is the upper
// half of a float, so the roundings come back by a shift and a mask
__device__ __forceinline__ uint32_t pack_remainder(float lo, float hi, uint32_t packed) {
  return pack(lo - __uint_as_float(packed << 16), hi - __uint_as_float(packed & 0xffff0000u));
}
__device__ __forceinline__ uint32_t pack_remainder(float lo, float hi) { return pack_remainder(lo, hi, pack(lo, hi)); }
// 2^x by the special-function unit (results below the smallest normal number are zero; 2^-inf = 0)
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

}  // namespace mma
}  // namespace pih
