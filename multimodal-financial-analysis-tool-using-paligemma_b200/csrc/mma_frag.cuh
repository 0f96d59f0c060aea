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
// O^T = diag(corr) O^T + V^T P^T of one chunk of 16 keys.  va: this lane's value rows 2j, 2j + 1, 2j + 8, 2j + 9 (8 columns of
// every 64); w: the scaled weights of key r (w[0], w[1]: heads 2j, 2j + 1) and key r + 8 (w[2], w[3]).
template <typename T, int VB>
__device__ __forceinline__ void add_values(float (&acc)[VB][4][4], const uint4 (&va)[VB][4], float (&w)[4], const float (&corr)[2]) {
  uint32_t pb[3][2];                                          // three 16-bit terms of the weights, as B fragments
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    pb[n][0] = transpose_8x8(split_pair<T>(w[0], w[1]));
    pb[n][1] = transpose_8x8(split_pair<T>(w[2], w[3]));
  }
#pragma unroll
  for (int vb = 0; vb < VB; ++vb) {
    const uint32_t* w0 = reinterpret_cast<const uint32_t*>(&va[vb][0]);
    const uint32_t* w1 = reinterpret_cast<const uint32_t*>(&va[vb][1]);
    const uint32_t* w2 = reinterpret_cast<const uint32_t*>(&va[vb][2]);
    const uint32_t* w3 = reinterpret_cast<const uint32_t*>(&va[vb][3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // rows r and r + 8 of this product: columns 64 vb + 8 r + 2 i and + 1
      const uint32_t a0 = __byte_perm(w0[i], w1[i], 0x5410), a1 = __byte_perm(w0[i], w1[i], 0x7632);
      const uint32_t a2 = __byte_perm(w2[i], w3[i], 0x5410), a3 = __byte_perm(w2[i], w3[i], 0x7632);
      float (&o)[4] = acc[vb][i];
      o[0] *= corr[0]; o[1] *= corr[1]; o[2] *= corr[0]; o[3] *= corr[1];
#pragma unroll
      for (int n = 0; n < 3; ++n) mma_16816<T>(o, a0, a1, a2, a3, pb[n][0], pb[n][1]);
    }
  }
}
// The same in fp32 multiplications, key by key: an infinite value times a weight's zero or negative second term is NaN above,
// times the weight itself infinite.  Keys behind the chunk's last one are left out.  values(k): this lane's columns of key k.
template <typename T, int VB, bool OWN_ROWS = false, typename Row>    // OWN_ROWS: the kernel itself writes some of them
__device__ __forceinline__ void add_values_fp32(float (&acc)[VB][4][4], Row values, const float (&w)[4], const float (&corr)[2], int keys) {
#pragma unroll
  for (int vb = 0; vb < VB; ++vb)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float (&o)[4] = acc[vb][i];
      o[0] *= corr[0]; o[1] *= corr[1]; o[2] *= corr[0]; o[3] *= corr[1];
    }
#pragma unroll 1
  for (int k = 0; k < min(16, keys); ++k) {
    const int src = (k & 7) * 4 + (threadIdx.x & 3);
    const float a0 = __shfl_sync(0xffffffffu, w[0], src), a1 = __shfl_sync(0xffffffffu, w[1], src);
    const float b0 = __shfl_sync(0xffffffffu, w[2], src), b1 = __shfl_sync(0xffffffffu, w[3], src);
    const float p0 = k < 8 ? a0 : b0, p1 = k < 8 ? a1 : b1;
    const T* row = values(k);
#pragma unroll
    for (int vb = 0; vb < VB; ++vb) {
      float f[8];
      unpack<T>(OWN_ROWS ? __ldcg(reinterpret_cast<const uint4*>(row + vb * 64)) : ldg_cached(row + vb * 64), f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float (&o)[4] = acc[vb][i];
        o[0] = fmaf(p0, f[2 * i], o[0]); o[1] = fmaf(p1, f[2 * i], o[1]);
        o[2] = fmaf(p0, f[2 * i + 1], o[2]); o[3] = fmaf(p1, f[2 * i + 1], o[3]);
      }
    }
  }
}
// Whether a sum of the warp's accumulators is NaN: some value was (or became) one, or infinities of both signs meet.
template <int VB>
__device__ __forceinline__ bool any_nan(const float (&acc)[VB][4][4]) {
  float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int vb = 0; vb < VB; ++vb)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] += acc[vb][i][e];
  const float t = (s[0] + s[1]) + (s[2] + s[3]);
  return __any_sync(0xffffffffu, t != t);
}
// this lane's 8 columns of head h of a quad's pair, without the weights' factor
template <typename T>
__device__ __forceinline__ void store_acc(float* dst, const float (&a)[4][4], int h) {
  constexpr float f = 1.f / split_scale<T>();
  reinterpret_cast<float4*>(dst)[0] = make_float4(a[0][h] * f, a[0][h + 2] * f, a[1][h] * f, a[1][h + 2] * f);
  reinterpret_cast<float4*>(dst)[1] = make_float4(a[2][h] * f, a[2][h + 2] * f, a[3][h] * f, a[3][h + 2] * f);
}

}  // namespace pg
