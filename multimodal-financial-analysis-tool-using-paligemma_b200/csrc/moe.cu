// Mixture-of-experts feed-forward for token batches: router, grouping of the (token, expert) pairs by expert,
// grouped expert GEMMs and the weighted combination into the fp32 residual stream.
//
//   pg_moe_route    fp32 router logits, softmax over all routed outputs, top-k on (score + correction), weights =
//                   score * scale (not renormalised); optional per-token sigmoid gate of a shared expert
//   pg_moe_route_topk  fp32 router logits with a bias, top-k on the logits, weights = softmax over the chosen ones
//   pg_moe_sort     pairs whose expert index is < n_experts are grouped by expert (offsets, source rows, position of
//                   each pair); larger indices are identity experts and take no part in the GEMMs
//   pg_moe_table_sort  experts picked by token id from a table: the grouping of every such layer of a model in one launch
//   pg_moe_gemm     out[pos] = A[row(pos)] W_e^T for the pairs of every expert e, optionally with the SwiGLU pairing
//                   silu(A Wg^T) * (A Wu^T) of stacked [Wg; Wu] weights, or with max(A W^T, 0)^2
//   pg_moe_combine  x[t] += sum_k w_k * (k-th expert's output, or the token's own input for an identity expert)
//                           + gate[t] * shared[t]
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace pg {

// ------------------------------------------------------------------ router: one CTA per token
// The token's row sits in shared memory as fp32; warp w computes the logits of the routed outputs w, w + warps, ...
// (16-byte weight loads when the rows allow), then warp 0 does the softmax, the top-k and the weights.
template <typename T>
__device__ __forceinline__ float dot_smem(const float* __restrict__ hs, const T* __restrict__ wr, int D, int lane) {
  constexpr int V = Vec<T>::N;
  float acc = 0.f;
  if (D % V == 0 && (reinterpret_cast<uintptr_t>(wr) & 15) == 0) {
    for (int k = lane * V; k < D; k += 32 * V) {
      float f[V];
      unpack<T>(ldg_cached(wr + k), f);
#pragma unroll
      for (int i = 0; i < V; ++i) acc = fmaf(hs[k + i], f[i], acc);
    }
  } else {
    for (int k = lane; k < D; k += 32) acc = fmaf(hs[k], to_f<T>(wr[k]), acc);
  }
  return warp_sum(acc);
}

// One warp: softmax over a token's logits s[0 .. n_route), the `top` largest of score + correction, weights = score * scale.
template <typename T>
__device__ __forceinline__ void route_softmax_pick(float* __restrict__ s, float* __restrict__ c, const T* __restrict__ correction,
                                                   int32_t* __restrict__ topk_idx, float* __restrict__ topk_w, size_t t, int n_route,
                                                   int top, float scale, int lane) {
  float mx = -INFINITY;
  for (int e = lane; e < n_route; e += 32) mx = fmaxf(mx, s[e]);
  mx = warp_max(mx);
  float sum = 0.f;
  for (int e = lane; e < n_route; e += 32) sum += expf(s[e] - mx);
  sum = warp_sum(sum);
  __syncwarp();
  for (int e = lane; e < n_route; e += 32) {
    const float pr = expf(s[e] - mx) / sum;
    s[e] = pr;
    c[e] = pr + (correction ? to_f<T>(correction[e]) : 0.f);
  }
  __syncwarp();
  for (int k = 0; k < top; ++k) {
    unsigned long long best = 0ull;
    for (int e = lane; e < n_route; e += 32) {
      const unsigned long long key = argmax_key(c[e], (unsigned)e);
      best = key > best ? key : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
      best = other > best ? other : best;
    }
    const int e = (int)argmax_key_index(best);
    if (lane == 0) {
      topk_idx[(size_t)t * top + k] = e;
      topk_w[(size_t)t * top + k] = s[e] * scale;
      c[e] = -INFINITY;
    }
    __syncwarp();
  }
}

// One warp: the choice among a token's sigmoid scores s and choice scores c (experts in groups), as described below.
template <typename T>
__device__ __forceinline__ void route_grouped_pick(float* __restrict__ s, float* __restrict__ c, float* __restrict__ gs,
                                                   int32_t* __restrict__ topk_idx, float* __restrict__ topk_w, size_t t, int n_route,
                                                   int top, int n_groups, int keep, int lane) {
  if (n_groups > 1 && keep < n_groups) {
    const int gsz = n_route / n_groups;
    for (int g = lane; g < n_groups; g += 32) {
      float a = -INFINITY, b = -INFINITY;          // the two largest of the group
      for (int e = g * gsz; e < (g + 1) * gsz; ++e) {
        const float v = c[e];
        if (v > a) { b = a; a = v; } else if (v > b) { b = v; }
      }
      gs[g] = gsz > 1 ? a + b : a;
    }
    __syncwarp();
    // the `keep` best groups are marked +inf one after the other; the groups left unmarked lose their experts
    for (int k = 0; k < keep; ++k) {
      unsigned long long best = 0ull;
      for (int g = lane; g < n_groups; g += 32) {
        if (gs[g] == INFINITY) continue;
        const unsigned long long key = argmax_key(gs[g], (unsigned)g);
        best = key > best ? key : best;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
      }
      if (lane == 0) gs[argmax_key_index(best)] = INFINITY;
      __syncwarp();
    }
    for (int e = lane; e < n_route; e += 32)
      if (gs[e / gsz] != INFINITY) c[e] = -INFINITY;
    __syncwarp();
  }
  float wsum = 0.f;
  for (int k = 0; k < top; ++k) {
    unsigned long long best = 0ull;
    for (int e = lane; e < n_route; e += 32) {
      if (s[e] < 0.f) continue;                    // chosen already (scores are sigmoids: never negative otherwise)
      const unsigned long long key = argmax_key(c[e], (unsigned)e);
      best = key > best ? key : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
      best = other > best ? other : best;
    }
    const int e = (int)argmax_key_index(best);
    const float se = s[e];
    wsum += se;
    __syncwarp();
    if (lane == 0) {
      topk_idx[(size_t)t * top + k] = e;
      topk_w[(size_t)t * top + k] = se;
      s[e] = -1.f;
    }
    __syncwarp();
  }
  const float inv = 1.f / (wsum + 1e-20f);
  for (int k = lane; k < top; k += 32) topk_w[(size_t)t * top + k] *= inv;
}

template <typename T>
__global__ void moe_route_kernel(int32_t* __restrict__ topk_idx, float* __restrict__ topk_w,
                                 float* __restrict__ shared_gate, const T* __restrict__ h, int ldh,
                                 const T* __restrict__ w_router, const T* __restrict__ correction,
                                 const T* __restrict__ w_sg, int T_, int D, int n_route, int top, float scale) {
  extern __shared__ float smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int t = blockIdx.x;
  float* hs = smem;                               // [D]
  float* s = smem + D;                            // scores [n_route]
  float* c = s + n_route;                         // choice scores [n_route]
  const T* hr = h + (size_t)t * ldh;
  for (int k = threadIdx.x; k < D; k += blockDim.x) hs[k] = to_f<T>(hr[k]);
  __syncthreads();
  for (int e = warp; e < n_route + 1; e += warps) {
    if (e < n_route) {
      const float z = dot_smem<T>(hs, w_router + (size_t)e * D, D, lane);
      if (lane == 0) s[e] = z;
    } else if (w_sg && shared_gate) {
      const float z = dot_smem<T>(hs, w_sg, D, lane);
      if (lane == 0) shared_gate[t] = 1.f / (1.f + expf(-z));
    }
  }
  __syncthreads();
  if (warp != 0) return;
  route_softmax_pick<T>(s, c, correction, topk_idx, topk_w, (size_t)t, n_route, top, scale, lane);
}

// ------------------------------------------------------------------ router with sigmoid scores and expert groups: one CTA per token
// z = h W_router^T in fp32, s = sigmoid(z); the choice scores are c = s + correction.  The experts form n_groups equal
// groups of neighbours; a group's score is the sum of its two largest choice scores (of the one, for groups of one),
// and only the experts of the `keep` best groups can be chosen (the others' choice scores count as -inf).  The `top`
// largest choice scores are chosen (ties: lowest index); the weights are the chosen s (without the correction)
// divided by their sum + 1e-20.
template <typename T>
__global__ void moe_route_grouped_kernel(int32_t* __restrict__ topk_idx, float* __restrict__ topk_w,
                                         const T* __restrict__ h, int ldh, const T* __restrict__ w_router,
                                         const T* __restrict__ correction, int T_, int D, int n_route, int top,
                                         int n_groups, int keep) {
  extern __shared__ float smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int t = blockIdx.x;
  float* hs = smem;                               // [D]
  float* s = smem + D;                            // scores [n_route]
  float* c = s + n_route;                         // choice scores [n_route]
  float* gs = c + n_route;                        // group scores [n_groups]
  const T* hr = h + (size_t)t * ldh;
  for (int k = threadIdx.x; k < D; k += blockDim.x) hs[k] = to_f<T>(hr[k]);
  __syncthreads();
  for (int e = warp; e < n_route; e += warps) {
    const float z = dot_smem<T>(hs, w_router + (size_t)e * D, D, lane);
    if (lane == 0) {
      const float sc = 1.f / (1.f + expf(-z));
      s[e] = sc;
      c[e] = sc + (correction ? to_f<T>(correction[e]) : 0.f);
    }
  }
  __syncthreads();
  if (warp != 0) return;
  route_grouped_pick<T>(s, c, gs, topk_idx, topk_w, (size_t)t, n_route, top, n_groups, keep, lane);
}

// ------------------------------------------------------------------ both routers over many tokens
// A CTA per token reads the whole router matrix for one row (8192 tokens x 16 experts x 2048 columns: 133 us, the router rows
// out of L1 / L2 once per token).  Here a warp takes RT_TOK tokens and RT_E router rows at a time: a 16-byte load of a router
// row feeds RT_TOK * 8 FMAs out of registers, the RT_TOK * RT_E = 32 lane partials meet in a transposed butterfly (31 shuffles
// leave lane L with the sum of pair L).  All loads of a step go out together (with a branch per router row in front of its
// load the same size took 82 us): that size runs in 36 us.  Products and sums stay fp32.
constexpr int RT_TOK = 4, RT_E = 8, RT_WARPS = 4;

template <typename T, bool GROUPED>
__global__ void __launch_bounds__(RT_WARPS * 32)
moe_route_tile_kernel(int32_t* __restrict__ topk_idx, float* __restrict__ topk_w, float* __restrict__ shared_gate,
                      const T* __restrict__ h, int ldh, const T* __restrict__ w_router, const T* __restrict__ correction,
                      const T* __restrict__ w_sg, int n_tokens, int D, int n_route, int top, float scale, int n_groups, int keep) {
  extern __shared__ float smem[];
  constexpr int V = Vec<T>::N;
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = (blockIdx.x * RT_WARPS + warp) * RT_TOK;
  if (t0 >= n_tokens) return;                     // nothing below waits for another warp
  const int nt = min(RT_TOK, n_tokens - t0);
  const int per_tok = 2 * n_route + (GROUPED ? n_groups : 0);
  float* st = smem + (size_t)warp * RT_TOK * per_tok;      // per token: scores, choice scores (, group scores)
  const T* hr[RT_TOK];
#pragma unroll
  for (int i = 0; i < RT_TOK; ++i) hr[i] = h + (size_t)(t0 + min(i, nt - 1)) * ldh;
  const int rows = n_route + (!GROUPED && w_sg && shared_gate ? 1 : 0);
  for (int e0 = 0; e0 < rows; e0 += RT_E) {
    float acc[RT_TOK * RT_E];
#pragma unroll
    for (int i = 0; i < RT_TOK * RT_E; ++i) acc[i] = 0.f;
    const T* wr[RT_E];                            // rows behind the last one repeat it; nobody reads their sums
#pragma unroll
    for (int e = 0; e < RT_E; ++e) {
      const int r = min(e0 + e, rows - 1);
      wr[e] = r < n_route ? w_router + (size_t)r * D : w_sg;
    }
    for (int k = lane * V; k < D; k += 32 * V) {
      uint4 xv[RT_TOK], wv[RT_E];                 // all loads of the step in flight together
#pragma unroll
      for (int i = 0; i < RT_TOK; ++i) xv[i] = ldg_cached(hr[i] + k);
#pragma unroll
      for (int e = 0; e < RT_E; ++e) wv[e] = ldg_cached(wr[e] + k);
      float x[RT_TOK][V];
#pragma unroll
      for (int i = 0; i < RT_TOK; ++i) unpack<T>(xv[i], x[i]);
#pragma unroll
      for (int e = 0; e < RT_E; ++e) {
        float f[V];
        unpack<T>(wv[e], f);
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
          for (int i = 0; i < RT_TOK; ++i) acc[i * RT_E + e] = fmaf(x[i][v], f[v], acc[i * RT_E + e]);
      }
    }
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
      const bool up = (lane & w) != 0;
#pragma unroll
      for (int i = 0; i < w; ++i) {
        const float keep_v = up ? acc[i + w] : acc[i];
        const float send = up ? acc[i] : acc[i + w];
        acc[i] = keep_v + __shfl_xor_sync(0xffffffffu, send, w);
      }
    }
    const int i = lane / RT_E, e = e0 + lane % RT_E;
    const float z = acc[0];
    if (i < nt && e < n_route) {
      float* s = st + i * per_tok;
      if (GROUPED) {
        const float sc = 1.f / (1.f + expf(-z));
        s[e] = sc;
        s[n_route + e] = sc + (correction ? to_f<T>(correction[e]) : 0.f);
      } else {
        s[e] = z;
      }
    } else if (i < nt && e == n_route && e < rows) {
      shared_gate[t0 + i] = 1.f / (1.f + expf(-z));
    }
  }
  __syncwarp();
  for (int i = 0; i < nt; ++i) {
    float* s = st + i * per_tok;
    if (GROUPED) route_grouped_pick<T>(s, s + n_route, s + 2 * n_route, topk_idx, topk_w, (size_t)(t0 + i), n_route, top, n_groups, keep, lane);
    else route_softmax_pick<T>(s, s + n_route, correction, topk_idx, topk_w, (size_t)(t0 + i), n_route, top, scale, lane);
  }
}

// The tile kernel takes 16-byte loads of both operands and pays where its warps fill the chip (16 tokens a CTA) or a CTA per token
// reads the router often enough; its own time hardly depends on the tokens before the chip is full.  us, CTA per token against
// tile: 512 tokens, 16 experts, width 2048 12 : 20 (128 experts 63 : 94), 1024 tokens 23 : 20 (124 : 93), 4 experts 9 : 12, 3072
// tokens 54 : 34 (303 : 137).  `line`: experts x width from which 1024 tokens are enough.
template <typename T>
static bool route_tile_wanted(const void* h, int ldh, const void* w_router, const void* w_sg, int n_tokens, int D, int n_route, int line,
                              size_t smem) {
  constexpr int V = Vec<T>::N;
  return (n_tokens >= 3072 || (n_tokens >= 1024 && (long long)n_route * D >= line)) && D % V == 0 && ldh % V == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(w_router) & 15) == 0 && (reinterpret_cast<uintptr_t>(w_sg) & 15) == 0 && smem <= 96 * 1024;
}

// Warps of a CTA per token.  A warp per routed output is one short chain for a few tokens; from about two CTAs per SM on it leaves
// fewer tokens side by side and the idle warps of the choice cost more (16 experts, width 2048: 256 tokens 7 us, 8 warps 12;
// 32 experts: 13 and 19; 768 tokens 34 and 23).
static int route_warps(int n_tokens, int outputs) { return max(4, min(n_tokens <= 256 ? 32 : 8, outputs)); }

// ------------------------------------------------------------------ router whose weights are a softmax over the chosen logits
// z = h W_router^T + bias in fp32; the `top` largest z are chosen (ties: lowest index) and weighted by the softmax over the
// chosen z alone.  A CTA serves TOK tokens: a warp takes an expert and streams its router row once for all of them.
// With `logits` (fp32 [n_tokens][n_route], before the bias: a GEMM of the step left them) only the choice is made here.
template <typename T, int TOK>
__global__ void __launch_bounds__(512)
moe_route_topk_kernel(int32_t* __restrict__ topk_idx, float* __restrict__ topk_w, const float* __restrict__ logits,
                      const T* __restrict__ h, int ldh,
                      const T* __restrict__ w_router, const T* __restrict__ bias, int n_tokens, int D, int n_route, int top) {
  extern __shared__ float smem[];
  float* hs = smem;                               // [TOK][D]
  float* z = logits ? smem : smem + TOK * D;      // [TOK][n_route]
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int t0 = blockIdx.x * TOK, nt = min(TOK, n_tokens - t0);
  constexpr int V = Vec<T>::N;
  const bool vec = D % V == 0 && (reinterpret_cast<uintptr_t>(w_router) & 15) == 0;
  if (logits) {
    for (int i = threadIdx.x; i < nt * n_route; i += blockDim.x)
      z[i] = logits[(size_t)t0 * n_route + i] + (bias ? to_f<T>(bias[i % n_route]) : 0.f);
  } else if (vec && ldh % V == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0) {
    for (int i = threadIdx.x * V; i < TOK * D; i += blockDim.x * V) {
      const int tt = i / D, k = i - tt * D;
      float f[V];
#pragma unroll
      for (int q = 0; q < V; ++q) f[q] = 0.f;
      if (tt < nt) unpack<T>(*reinterpret_cast<const uint4*>(h + (size_t)(t0 + tt) * ldh + k), f);
#pragma unroll
      for (int q = 0; q < V; ++q) hs[i + q] = f[q];
    }
  } else {
    for (int i = threadIdx.x; i < TOK * D; i += blockDim.x) {
      const int tt = i / D;
      hs[i] = tt < nt ? to_f<T>(h[(size_t)(t0 + tt) * ldh + i - tt * D]) : 0.f;
    }
  }
  __syncthreads();
  for (int e = warp; !logits && e < n_route; e += warps) {
    const T* wr = w_router + (size_t)e * D;
    float acc[TOK];
#pragma unroll
    for (int tt = 0; tt < TOK; ++tt) acc[tt] = 0.f;
    if (vec) {
      for (int k = lane * V; k < D; k += 32 * V) {
        float f[V];
        unpack<T>(ldg_cached(wr + k), f);
#pragma unroll
        for (int tt = 0; tt < TOK; ++tt)
#pragma unroll
          for (int q = 0; q < V; q += 4) {
            const float4 x = *reinterpret_cast<const float4*>(hs + tt * D + k + q);
            acc[tt] = fmaf(x.x, f[q], acc[tt]); acc[tt] = fmaf(x.y, f[q + 1], acc[tt]);
            acc[tt] = fmaf(x.z, f[q + 2], acc[tt]); acc[tt] = fmaf(x.w, f[q + 3], acc[tt]);
          }
      }
    } else {
      for (int k = lane; k < D; k += 32) {
        const float f = to_f<T>(wr[k]);
#pragma unroll
        for (int tt = 0; tt < TOK; ++tt) acc[tt] = fmaf(hs[tt * D + k], f, acc[tt]);
      }
    }
    const float b = bias ? to_f<T>(bias[e]) : 0.f;
#pragma unroll
    for (int tt = 0; tt < TOK; ++tt) {
      const float v = warp_sum(acc[tt]);
      if (lane == 0) z[tt * n_route + e] = v + b;
    }
  }
  __syncthreads();
  for (int tt = warp; tt < nt; tt += warps) {      // a warp per token: top-k, then the weights
    float* zt = z + tt * n_route;
    const size_t o = (size_t)(t0 + tt) * top;
    float z0 = 0.f, sum = 0.f;
    for (int k = 0; k < top; ++k) {
      unsigned long long best = 0ull;
      for (int e = lane; e < n_route; e += 32) {
        const unsigned long long key = argmax_key(zt[e], (unsigned)e);
        best = key > best ? key : best;
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, s);
        best = other > best ? other : best;
      }
      const int e = (int)argmax_key_index(best);
      const float v = argmax_key_value(best);
      if (k == 0) z0 = v;
      const float w = expf(v - z0);
      sum += w;
      __syncwarp();
      if (lane == 0) { topk_idx[o + k] = e; topk_w[o + k] = w; zt[e] = -INFINITY; }
      __syncwarp();
    }
    const float inv = 1.f / sum;
    for (int k = lane; k < top; k += 32) topk_w[o + k] *= inv;
  }
}

// ------------------------------------------------------------------ group the pairs by expert (one cluster)
// A cluster of `CTAs` (1 or 8) takes the pairs in equal consecutive parts.  One shared-memory atomic per pair counts it and gives
// its place among its CTA's pairs of the expert; the CTAs read each other's counts through distributed shared memory for the
// first position of every (expert, CTA).  One CTA alone is bound by its own atomics and scattered stores: 16384 pairs of 16
// experts 15.1 us (16.4 with one atomic per pair on eight counters per expert, 22.9 with lanes grouped by match.any),
// this 6.7 us with eight.
constexpr int SORT_ITEMS = 16, SORT_CTAS = 8, SORT_THREADS = 256;

__global__ void __launch_bounds__(SORT_THREADS)
moe_sort_kernel(int32_t* __restrict__ offsets, int32_t* __restrict__ sorted_row, int32_t* __restrict__ pair_pos,
                const int32_t* __restrict__ topk_idx, int n_pairs, int top, int n_experts) {
  extern __shared__ int sm_i[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = (int)gridDim.x, rank = (int)blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  int* count = sm_i;                   // [n_experts]: this CTA's pairs of an expert (read by the other CTAs)
  int* first = sm_i + n_experts;       // [n_experts]: position of the first of them
  for (int e = threadIdx.x; e < n_experts; e += SORT_THREADS) count[e] = 0;
  __syncthreads();
  constexpr int ROUND = SORT_ITEMS * SORT_THREADS;
  const int per = (n_pairs + ctas - 1) / ctas, begin = rank * per, end = min(n_pairs, begin + per);
  const bool one_round = per <= ROUND;
  int ex[SORT_ITEMS], place[SORT_ITEMS];
  for (int i0 = begin; i0 < end; i0 += ROUND) {
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; ++k) {          // a round's loads are in flight together
      const int i = i0 + k * SORT_THREADS + threadIdx.x;
      const int e = i < end ? topk_idx[i] : -1;
      ex[k] = e >= 0 && e < n_experts ? e : -1;     // -1: no place in the grouped order
    }
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; ++k) {
      const int i = i0 + k * SORT_THREADS + threadIdx.x;
      place[k] = ex[k] >= 0 ? atomicAdd(&count[ex[k]], 1) : -1;
      if (!one_round && i < end) pair_pos[i] = place[k];   // this thread takes it up again below
    }
  }
  if (ctas > 1) cluster.sync(); else __syncthreads();    // every CTA's counts are complete
  if (threadIdx.x < 32) {              // prefix over the experts, 32 at a time, and over the CTAs inside an expert
    const int lane = threadIdx.x;
    int base = 0;
    for (int e0 = 0; e0 < n_experts; e0 += 32) {
      int total = 0, before = 0;
      if (e0 + lane < n_experts)
        for (int c = 0; c < ctas; ++c) {
          const int n = ctas > 1 ? *cluster.map_shared_rank(count + e0 + lane, c) : count[e0 + lane];
          total += n;
          if (c < rank) before += n;
        }
      int inc = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += v; }
      if (e0 + lane < n_experts) {
        first[e0 + lane] = base + inc - total + before;
        if (rank == 0) offsets[e0 + lane] = base + inc - total;
      }
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (rank == 0 && lane == 0) offsets[n_experts] = base;
  }
  if (ctas > 1) cluster.sync(); else __syncthreads();    // `first` is there; nobody reads another CTA's counts any more
  // the order of the pairs inside a group does not change any result: every output row is computed on its own
  for (int i0 = begin; i0 < end; i0 += ROUND) {
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; ++k) {
      const int i = i0 + k * SORT_THREADS + threadIdx.x;
      if (i >= end) break;
      if (!one_round) {
        place[k] = pair_pos[i];
        ex[k] = place[k] >= 0 ? topk_idx[i] : -1;
      }
      const int pos = place[k] >= 0 ? first[ex[k]] + place[k] : -1;
      if (pos >= 0) sorted_row[pos] = i / top;
      pair_pos[i] = pos;
    }
  }
}

// ------------------------------------------------------------------ experts picked by token id: every layer's grouping at once
// Routing by a table [vocab, top] of expert indices depends on the token ids alone, so the pairs of ALL such layers are
// grouped before the first layer runs: CTA l handles layer l.  desc[l] = {first entry of the layer's table in `tables`,
// experts, top, sum of the earlier layers' top, sum of the earlier layers' (experts + 1)}.  Layer l's pair_pos starts at
// n_tokens * desc[l][3], its offsets at desc[l][4].  An id outside the vocabulary gets no place (-1).
__global__ void __launch_bounds__(1024)
moe_table_sort_kernel(int32_t* __restrict__ offsets, int32_t* __restrict__ pair_pos, const int32_t* __restrict__ tables,
                      const int32_t* __restrict__ desc, const int64_t* __restrict__ ids, int n_tokens, long long vocab,
                      int max_experts) {
  extern __shared__ int sm_i[];
  pdl_launch_dependents();
  pdl_wait();
  const int32_t* d = desc + 5 * blockIdx.x;
  const int E = d[1], top = d[2];
  const int32_t* table = tables + d[0];
  int32_t* pos = pair_pos + (size_t)n_tokens * d[3];
  int32_t* off = offsets + d[4];
  int* count = sm_i;                   // [max_experts]
  int* cursor = sm_i + max_experts;    // [max_experts]
  for (int e = threadIdx.x; e < E; e += blockDim.x) count[e] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, n_pairs = n_tokens * top, round = SORT_ITEMS * blockDim.x;
  int ex[SORT_ITEMS];                  // a round's experts of this thread: all its loads are in flight together
  auto load_round = [&](int i0) {
    int64_t id[SORT_ITEMS];
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; ++k) {
      const int i = i0 + k * blockDim.x + threadIdx.x;
      id[k] = i < n_pairs ? ids[i / top] : -1;
    }
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; ++k) {
      const int i = i0 + k * blockDim.x + threadIdx.x;
      const int e = (id[k] >= 0 && id[k] < vocab) ? table[id[k] * top + i % top] : -1;
      ex[k] = e < E ? e : -1;
    }
  };
  for (int i0 = 0; i0 < n_pairs; i0 += round) {
    load_round(i0);
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; ++k)
      if (ex[k] >= 0) atomicAdd(&count[ex[k]], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {              // exclusive prefix over the experts, 32 at a time
    int base = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int c = e0 + lane < E ? count[e0 + lane] : 0;
      int inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += v; }
      if (e0 + lane < E) { off[e0 + lane] = base + inc - c; cursor[e0 + lane] = base + inc - c; }
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) off[E] = base;
  }
  __syncthreads();
  // the order of the pairs inside a group does not change any result: every output row is computed on its own
  for (int i0 = 0; i0 < n_pairs; i0 += round) {
    if (n_pairs > round) load_round(i0);            // a single round is still in registers
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; ++k) {
      const int i = i0 + k * blockDim.x + threadIdx.x;
      if (i < n_pairs) pos[i] = ex[k] >= 0 ? atomicAdd(&cursor[ex[k]], 1) : -1;
    }
  }
}

// ------------------------------------------------------------------ grouped GEMM, fp32 FMA (any dtype)
// The gated pairings of a stacked [Wg; Wu] product (g, u already rounded to the model dtype):
//   PG_GLU_SILU    silu(g) * u
//   PG_GLU_CLAMPED g' = min(g, limit), u' = clamp(u, -limit, limit): g' sigmoid(1.702 g') (u' + 1)
template <typename T>
__device__ __forceinline__ float glu_pair(float g, float u, int act, float limit) {
  if (act == PG_GLU_CLAMPED) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return rnd<T>(g / (1.f + expf(-1.702f * g))) * (u + 1.f);
  }
  return rnd<T>(rnd<T>(g / (1.f + expf(-g))) * u);
}

constexpr int MG_BM = 64, MG_BN = 64, MG_BK = 16, MG_THREADS = 256, MG_PAD = 4;

template <typename T, bool DUAL>
__global__ void __launch_bounds__(MG_THREADS)
moe_gemm_simt_kernel(T* __restrict__ out, int ldo, const T* __restrict__ A, int lda,
                     const int32_t* __restrict__ row_map, const T* __restrict__ W,
                     const int32_t* __restrict__ offsets, int n_experts, int N, int K, int act, float limit) {
  __shared__ __align__(16) float As[MG_BK][MG_BM + MG_PAD];
  __shared__ __align__(16) float Bs[MG_BK][MG_BN + MG_PAD];
  __shared__ __align__(16) float Us[DUAL ? MG_BK : 1][MG_BN + MG_PAD];
  __shared__ int s_tile[3];
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0) {
    int tile = blockIdx.y, e = 0, acc = 0;
    for (; e < n_experts; ++e) {
      const int nt = (offsets[e + 1] - offsets[e] + MG_BM - 1) / MG_BM;
      if (tile < acc + nt) break;
      acc += nt;
    }
    s_tile[0] = e;
    s_tile[1] = e < n_experts ? offsets[e] + (tile - acc) * MG_BM : 0;
    s_tile[2] = e < n_experts ? offsets[e + 1] : 0;
  }
  __syncthreads();
  const int e = s_tile[0], m0 = s_tile[1], m_end = s_tile[2];
  if (e >= n_experts) return;
  const int n0 = blockIdx.x * MG_BN;
  const int n_w = DUAL ? 2 * N : N;
  const T* We = W + (size_t)e * n_w * K;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float acc[4][4], acu[DUAL ? 4 : 1][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[i][j] = 0.f; if (DUAL) acu[i][j] = 0.f; }
  for (int k0 = 0; k0 < K; k0 += MG_BK) {
    for (int idx = threadIdx.x; idx < MG_BM * MG_BK; idx += MG_THREADS) {
      const int r = idx / MG_BK, kk = idx % MG_BK;
      float a = 0.f, b = 0.f, u = 0.f;
      if (k0 + kk < K) {
        if (m0 + r < m_end) {
          const int src = row_map ? row_map[m0 + r] : m0 + r;
          a = to_f<T>(A[(size_t)src * lda + k0 + kk]);
        }
        if (n0 + r < N) {
          b = to_f<T>(We[(size_t)(n0 + r) * K + k0 + kk]);
          if (DUAL) u = to_f<T>(We[(size_t)(N + n0 + r) * K + k0 + kk]);
        }
      }
      As[kk][r] = a;
      Bs[kk][r] = b;
      if (DUAL) Us[kk][r] = u;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < MG_BK; ++kk) {
      const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      if (DUAL) {
        const float4 u = *reinterpret_cast<const float4*>(&Us[kk][tx * 4]);
        const float uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acu[i][j] = fmaf(av[i], uv[j], acu[i][j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= m_end) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = act == PG_ACT_RELU2 ? fmaxf(acc[i][j], 0.f) : rnd<T>(acc[i][j]);
      if (act == PG_ACT_RELU2) v *= v;
      if (DUAL) v = glu_pair<T>(v, rnd<T>(acu[DUAL ? i : 0][j]), act, limit);
      out[(size_t)m * ldo + n] = from_f<T>(v);
    }
  }
}

// ------------------------------------------------------------------ weighted combination into the residual stream
template <typename T>
__global__ void moe_combine_kernel(float* __restrict__ x, T* __restrict__ out, int ldo, const T* __restrict__ y, int ldy,
                                   const int32_t* __restrict__ pair_pos, const float* __restrict__ topk_w,
                                   const T* __restrict__ h, int ldh, const T* __restrict__ shared_out, int lds,
                                   const float* __restrict__ shared_gate, int D, int top) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    float acc = 0.f;
    for (int k = 0; k < top; ++k) {
      const int pos = pair_pos[(size_t)t * top + k];
      const float w = topk_w[(size_t)t * top + k];
      const float v = pos >= 0 ? to_f<T>(y[(size_t)pos * ldy + c]) : to_f<T>(h[(size_t)t * ldh + c]);
      acc = fmaf(w, v, acc);
    }
    if (shared_out) acc = fmaf(shared_gate ? shared_gate[t] : 1.f, to_f<T>(shared_out[(size_t)t * lds + c]), acc);
    if (out) out[(size_t)t * ldo + c] = from_f<T>(acc);
    else x[(size_t)t * D + c] += acc;
  }
}

// 16 bytes of a row per thread, the rows of a token's experts requested COMBINE_K at a time: 8192 tokens x 2 rows x 2048
// columns in 23 us, near the copy rate (an element per thread and load: 55 us).  Sums run in the order of k.
constexpr int COMBINE_K = 4;

template <typename T>
__global__ void __launch_bounds__(256)
moe_combine_vec_kernel(float* __restrict__ x, T* __restrict__ out, int ldo, const T* __restrict__ y, int ldy,
                       const int32_t* __restrict__ pair_pos, const float* __restrict__ topk_w, const T* __restrict__ h, int ldh,
                       const T* __restrict__ shared_out, int lds, const float* __restrict__ shared_gate, int D, int top) {
  constexpr int V = Vec<T>::N;
  pdl_launch_dependents();
  pdl_wait();
  const size_t t = blockIdx.x;
  const float sg = shared_out && shared_gate ? shared_gate[t] : 1.f;
  for (int c = threadIdx.x * V; c < D; c += blockDim.x * V) {
    float acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.f;
    uint4 so = make_uint4(0, 0, 0, 0);
    if (shared_out) so = ldg_cached(shared_out + t * lds + c);
    for (int k0 = 0; k0 < top; k0 += COMBINE_K) {
      uint4 r[COMBINE_K];
      float w[COMBINE_K];
#pragma unroll
      for (int k = 0; k < COMBINE_K; ++k) {
        if (k0 + k < top) {
          const int pos = pair_pos[t * top + k0 + k];
          w[k] = topk_w[t * top + k0 + k];
          r[k] = ldg_cached(pos >= 0 ? y + (size_t)pos * ldy + c : h + t * ldh + c);
        }
      }
#pragma unroll
      for (int k = 0; k < COMBINE_K; ++k) {
        if (k0 + k < top) {
          float f[V];
          unpack<T>(r[k], f);
#pragma unroll
          for (int i = 0; i < V; ++i) acc[i] = fmaf(w[k], f[i], acc[i]);
        }
      }
    }
    if (shared_out) {
      float f[V];
      unpack<T>(so, f);
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = fmaf(sg, f[i], acc[i]);
    }
    if (out) {
      *reinterpret_cast<uint4*>(out + t * ldo + c) = pack<T>(acc);
    } else {
      float4* xr = reinterpret_cast<float4*>(x + t * D + c);
#pragma unroll
      for (int i = 0; i < V; i += 4) {
        float4 v = xr[i / 4];
        v.x += acc[i]; v.y += acc[i + 1]; v.z += acc[i + 2]; v.w += acc[i + 3];
        xr[i / 4] = v;
      }
    }
  }
}

// rows of the grouped order: out[pos] = a[row_map[pos]] (16-byte copies when the rows allow, else elements)
template <typename T>
__global__ void gather_rows_kernel(T* __restrict__ out, const T* __restrict__ a, int lda,
                                   const int32_t* __restrict__ row_map, const int32_t* __restrict__ n_rows, int cols) {
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.x;
  if (n_rows && r >= *n_rows) return;
  const T* src = a + (size_t)row_map[r] * lda;
  T* dst = out + (size_t)r * cols;
  constexpr int V = Vec<T>::N;
  if (cols % V == 0 && lda % V == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    for (int c = threadIdx.x * V; c < cols; c += blockDim.x * V)
      *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(src + c);
  } else {
    for (int c = threadIdx.x; c < cols; c += blockDim.x) dst[c] = src[c];
  }
}

int moe_gemm_tc(void* out, int ldo, const void* A, int lda, const int32_t* row_map, const void* W,
                const int32_t* offsets, int n_pairs, int n_experts, int N, int K, int act, float limit, int dtype,
                int* err_flag, cudaStream_t st);
bool moe_gemm_tc_supported(int ldo, int lda, const int32_t* row_map, int N, int K, int dtype);

}  // namespace pg

using namespace pg;

extern "C" int pg_moe_route(int32_t* topk_idx, float* topk_w, float* shared_gate, const void* h, int ldh,
                            const void* w_router, const void* correction, const void* w_shared_gate, int n_tokens,
                            int D, int n_route, int top, float scale, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(top >= 1 && top <= n_route && n_route <= 4096, "moe_route: top %d of %d routed outputs", top, n_route);
  const int warps = route_warps(n_tokens, n_route + 1);
  const size_t smem = sizeof(float) * ((size_t)D + 2 * (size_t)n_route);
  PG_REQUIRE(smem <= 200 * 1024, "moe_route: D=%d with %d routed outputs does not fit shared memory", D, n_route);
  PG_DISPATCH_DTYPE(dtype, T, {
    const size_t tile_smem = sizeof(float) * (size_t)RT_WARPS * RT_TOK * 2 * n_route;
    if (route_tile_wanted<T>(h, ldh, w_router, w_shared_gate, n_tokens, D, n_route, 32768, tile_smem))
      return launch_pdl("moe_route", moe_route_tile_kernel<T, false>, dim3(cdiv(n_tokens, RT_WARPS * RT_TOK)), dim3(RT_WARPS * 32),
                        tile_smem, (cudaStream_t)stream, topk_idx, topk_w, shared_gate, (const T*)h, ldh, (const T*)w_router,
                        (const T*)correction, (const T*)w_shared_gate, n_tokens, D, n_route, top, scale, 1, 1);
    auto kern = moe_route_kernel<T>;
    return launch_pdl("moe_route", kern, dim3(n_tokens), dim3(warps * 32), smem, (cudaStream_t)stream, topk_idx, topk_w,
                      shared_gate, (const T*)h, ldh, (const T*)w_router, (const T*)correction, (const T*)w_shared_gate,
                      n_tokens, D, n_route, top, scale);
  });
  return PG_OK;
}

extern "C" int pg_moe_sort(int32_t* offsets, int32_t* sorted_row, int32_t* pair_pos, const int32_t* topk_idx,
                           int n_pairs, int top, int n_experts, void* stream) {
  PG_REQUIRE(n_experts >= 1 && n_experts <= 4096 && top >= 1, "moe_sort: %d experts, top %d", n_experts, top);
  // eight CTAs from the count on at which one would walk several pairs per thread
  const int ctas = n_pairs > 4 * SORT_THREADS ? SORT_CTAS : 1;
  if (ctas == 1)
    return launch_pdl("moe_sort", moe_sort_kernel, dim3(1), dim3(SORT_THREADS), sizeof(int) * 2 * (size_t)n_experts,
                      (cudaStream_t)stream, offsets, sorted_row, pair_pos, topk_idx, n_pairs, top, n_experts);
  static const int pdl = env_int("PG_PDL", 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(SORT_THREADS);
  cfg.dynamicSmemBytes = sizeof(int) * 2 * (size_t)n_experts;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, moe_sort_kernel, offsets, sorted_row, pair_pos, topk_idx, n_pairs, top, n_experts);
  if (err != cudaSuccess) {
    set_error("moe_sort launch: %s", cudaGetErrorString(err));
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  return check_launch("moe_sort");
}

extern "C" int pg_moe_table_sort(int32_t* offsets, int32_t* pair_pos, const int32_t* tables, const int32_t* desc, int n_layers,
                                 const int64_t* ids, int n_tokens, long long vocab, int max_experts, void* stream) {
  if (n_layers <= 0 || n_tokens <= 0) return PG_OK;
  PG_REQUIRE(offsets && pair_pos && tables && desc && ids && max_experts >= 1 && max_experts <= 4096,
             "moe_table_sort: %d layers, up to %d experts", n_layers, max_experts);
  return launch_pdl("moe_table_sort", moe_table_sort_kernel, dim3(n_layers), dim3(n_tokens <= 64 ? 128 : 1024),
                    sizeof(int) * 2 * (size_t)max_experts, (cudaStream_t)stream, offsets, pair_pos, tables, desc, ids, n_tokens,
                    vocab, max_experts);
}

extern "C" int pg_moe_gemm_act(void* out, int ldo, const void* A, int lda, const int32_t* row_map, const void* W,
                               const int32_t* offsets, int n_pairs, int n_experts, int N, int K, int act, float limit,
                               int impl, int* err_flag, int dtype, void* stream) {
  if (n_pairs <= 0) return PG_OK;
  PG_REQUIRE(act == PG_GLU_NONE || act == PG_GLU_SILU || act == PG_GLU_CLAMPED || act == PG_ACT_RELU2,
             "moe_gemm: unknown pairing or activation %d", act);
  const int swiglu = act == PG_GLU_SILU || act == PG_GLU_CLAMPED;      // two products per output
  cudaStream_t st = (cudaStream_t)stream;
  if (impl != 1 && moe_gemm_tc_supported(ldo, lda, row_map, N, K, dtype))
    return moe_gemm_tc(out, ldo, A, lda, row_map, W, offsets, n_pairs, n_experts, N, K, act, limit, dtype, err_flag, st);
  PG_REQUIRE(impl != 2, "moe_gemm: the tensor-core kernel does not take this problem (N=%d K=%d dtype %d)", N, K, dtype);
  dim3 grid(cdiv(N, MG_BN), cdiv(n_pairs, MG_BM) + n_experts);
  PG_DISPATCH_DTYPE(dtype, T, {
    if (swiglu)
      return launch_pdl("moe_gemm", moe_gemm_simt_kernel<T, true>, grid, dim3(MG_THREADS), 0, st, (T*)out, ldo, (const T*)A,
                        lda, row_map, (const T*)W, offsets, n_experts, N, K, act, limit);
    return launch_pdl("moe_gemm", moe_gemm_simt_kernel<T, false>, grid, dim3(MG_THREADS), 0, st, (T*)out, ldo, (const T*)A,
                      lda, row_map, (const T*)W, offsets, n_experts, N, K, act, limit);
  });
  return PG_OK;
}

extern "C" int pg_moe_gemm(void* out, int ldo, const void* A, int lda, const int32_t* row_map, const void* W,
                           const int32_t* offsets, int n_pairs, int n_experts, int N, int K, int swiglu, int impl,
                           int* err_flag, int dtype, void* stream) {
  return pg_moe_gemm_act(out, ldo, A, lda, row_map, W, offsets, n_pairs, n_experts, N, K,
                         swiglu ? PG_GLU_SILU : PG_GLU_NONE, 0.f, impl, err_flag, dtype, stream);
}

extern "C" int pg_moe_route_grouped(int32_t* topk_idx, float* topk_w, const void* h, int ldh, const void* w_router,
                                    const void* correction, int n_tokens, int D, int n_route, int top, int n_groups,
                                    int keep, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(top >= 1 && top <= n_route && n_route <= 4096, "moe_route: top %d of %d routed outputs", top, n_route);
  PG_REQUIRE(n_groups >= 1 && n_route % n_groups == 0 && keep >= 1 && keep <= n_groups &&
                 (long long)keep * (n_route / n_groups) >= top,
             "moe_route: %d groups over %d experts, %d kept, top %d", n_groups, n_route, keep, top);
  const int warps = route_warps(n_tokens, n_route);
  const size_t smem = sizeof(float) * ((size_t)D + 2 * (size_t)n_route + n_groups);
  PG_REQUIRE(smem <= 200 * 1024, "moe_route: D=%d with %d routed outputs does not fit shared memory", D, n_route);
  PG_DISPATCH_DTYPE(dtype, T, {
    const size_t tile_smem = sizeof(float) * (size_t)RT_WARPS * RT_TOK * (2 * n_route + n_groups);
    if (route_tile_wanted<T>(h, ldh, w_router, nullptr, n_tokens, D, n_route, 65536, tile_smem))
      return launch_pdl("moe_route_grouped", moe_route_tile_kernel<T, true>, dim3(cdiv(n_tokens, RT_WARPS * RT_TOK)),
                        dim3(RT_WARPS * 32), tile_smem, (cudaStream_t)stream, topk_idx, topk_w, (float*)nullptr, (const T*)h, ldh,
                        (const T*)w_router, (const T*)correction, (const T*)nullptr, n_tokens, D, n_route, top, 1.f, n_groups, keep);
    auto kern = moe_route_grouped_kernel<T>;
    return launch_pdl("moe_route_grouped", kern, dim3(n_tokens), dim3(warps * 32), smem, (cudaStream_t)stream, topk_idx,
                      topk_w, (const T*)h, ldh, (const T*)w_router, (const T*)correction, n_tokens, D, n_route, top,
                      n_groups, keep);
  });
  return PG_OK;
}

extern "C" int pg_moe_route_topk(int32_t* topk_idx, float* topk_w, const float* logits, const void* h, int ldh, const void* w_router,
                                 const void* bias, int n_tokens, int D, int n_route, int top, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(topk_idx && topk_w && (logits || (h && w_router)) && top >= 1 && top <= n_route && n_route <= 4096,
             "moe_route_topk: top %d of %d routed outputs", top, n_route);
  auto smem = [&](int tok) { return sizeof(float) * (size_t)tok * ((logits ? 0 : (size_t)D) + n_route); };
  PG_REQUIRE(smem(1) <= 200 * 1024, "moe_route_topk: D=%d with %d routed outputs does not fit shared memory", D, n_route);
  PG_DISPATCH_DTYPE(dtype, T, {
    if (n_tokens >= 296 && smem(8) <= 100 * 1024)
      return launch_pdl("moe_route_topk", moe_route_topk_kernel<T, 8>, dim3(cdiv(n_tokens, 8)), dim3(256), smem(8), (cudaStream_t)stream,
                        topk_idx, topk_w, logits, (const T*)h, ldh, (const T*)w_router, (const T*)bias, n_tokens, D, n_route, top);
    return launch_pdl("moe_route_topk", moe_route_topk_kernel<T, 1>, dim3(n_tokens), dim3(n_route >= 16 && !logits ? 512 : 256), smem(1),
                      (cudaStream_t)stream, topk_idx, topk_w, logits, (const T*)h, ldh, (const T*)w_router, (const T*)bias, n_tokens,
                      D, n_route, top);
  });
  return PG_OK;
}

static int moe_combine_any(float* x, void* out, int ldo, const void* y, int ldy, const int32_t* pair_pos,
                           const float* topk_w, const void* h, int ldh, const void* shared_out, int lds,
                           const float* shared_gate, int n_tokens, int D, int top, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  auto fits = [](const void* p, long long ld, int vec) { return !p || (((uintptr_t)p & 15) == 0 && ld % vec == 0); };
  PG_DISPATCH_DTYPE(dtype, T, {
    constexpr int V = Vec<T>::N;
    if (D % V == 0 && fits(x, D, 4) && fits(out, ldo, V) && fits(y, ldy, V) && fits(h, ldh, V) && fits(shared_out, lds, V)) {
      const int vecs = D / V, threads = vecs >= 256 ? 256 : (vecs + 31) / 32 * 32;
      return launch_pdl("moe_combine", moe_combine_vec_kernel<T>, dim3(n_tokens), dim3(threads), 0, (cudaStream_t)stream, x,
                        (T*)out, ldo, (const T*)y, ldy, pair_pos, topk_w, (const T*)h, ldh, (const T*)shared_out, lds,
                        shared_gate, D, top);
    }
    const int threads = n_tokens <= 64 ? (D >= 2048 ? 512 : 256) : 128;
    return launch_pdl("moe_combine", moe_combine_kernel<T>, dim3(n_tokens), dim3(threads), 0, (cudaStream_t)stream, x,
                      (T*)out, ldo, (const T*)y, ldy, pair_pos, topk_w, (const T*)h, ldh, (const T*)shared_out, lds,
                      shared_gate, D, top);
  });
  return PG_OK;
}

extern "C" int pg_moe_combine(float* x, const void* y, int ldy, const int32_t* pair_pos, const float* topk_w,
                              const void* h, int ldh, const void* shared_out, int lds, const float* shared_gate,
                              int n_tokens, int D, int top, int dtype, void* stream) {
  return moe_combine_any(x, nullptr, 0, y, ldy, pair_pos, topk_w, h, ldh, shared_out, lds, shared_gate, n_tokens, D, top,
                         dtype, stream);
}

extern "C" int pg_moe_combine_out(void* out, int ldo, const void* y, int ldy, const int32_t* pair_pos,
                                  const float* topk_w, const void* shared_out, int lds, int n_tokens, int D, int top,
                                  int dtype, void* stream) {
  PG_REQUIRE(out && ldo >= D, "moe_combine_out: an output of %d columns", D);
  return moe_combine_any(nullptr, out, ldo, y, ldy, pair_pos, topk_w, nullptr, 0, shared_out, lds, nullptr, n_tokens, D,
                         top, dtype, stream);
}

extern "C" int pg_gather_rows(void* out, const void* a, int lda, const int32_t* row_map, const int32_t* n_rows,
                              int max_rows, int cols, int dtype, void* stream) {
  if (max_rows <= 0) return PG_OK;
  PG_DISPATCH_DTYPE(dtype, T, {
    return launch_pdl("gather_rows", gather_rows_kernel<T>, dim3(max_rows), dim3(128), 0, (cudaStream_t)stream, (T*)out,
                      (const T*)a, lda, row_map, n_rows, cols);
  });
  return PG_OK;
}
