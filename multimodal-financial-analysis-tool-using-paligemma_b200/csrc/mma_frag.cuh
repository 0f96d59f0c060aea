// mma.sync fragments of the decode attention kernels (16-bit operands, fp32 accumulation).
#pragma once
#include "common.cuh"

namespace pg {

template <typename T>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, bf16>::value)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
// fp32 weights enter a product as three 16-bit terms.  In bf16 (fp32's exponents) the terms hold all 24 bits.  An fp16 term
// resolves 2^-24 at best, so weights of at most 1 are multiplied by 2^14 first and the accumulators divided by it: what is
// left over is below 2^-39 of the largest weight, where an fp32 sum that this weight is part of rounds at 2^-24.  (Without the
// factor 4096 weights of 3e-7 beside one of 1 lost 2.6 % of their sum.)  Weights that nothing normalises do not go this way.
template <typename T>
constexpr float split_scale() { return std::is_same<T, bf16>::value ? 1.f : 16384.f; }
// (x, y) as two 16-bit values of T (x in the low half); x and y become what the rounding left over
template <typename T>
__device__ __forceinline__ uint32_t split_pair(float& x, float& y) {
  if constexpr (std::is_same<T, bf16>::value) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    x -= __low2float(h);
    y -= __high2float(h);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __half2 h = __floats2half2_rn(x, y);
    x -= __low2float(h);
    y -= __high2float(h);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}
// this lane's 8 columns of head h of a quad's pair, without the weights' factor
template <typename T>
__device__ __forceinline__ void store_acc(float* dst, const float (&a)[4][4], int h) {
  constexpr float f = 1.f / split_scale<T>();
  reinterpret_cast<float4*>(dst)[0] = make_float4(a[0][h] * f, a[0][h + 2] * f, a[1][h] * f, a[1][h + 2] * f);
  reinterpret_cast<float4*>(dst)[1] = make_float4(a[2][h] * f, a[2][h + 2] * f, a[3][h] * f, a[3][h + 2] * f);
}

}  // namespace pg
