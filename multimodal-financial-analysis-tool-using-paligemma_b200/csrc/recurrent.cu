// Recurrent mixers for ragged token batches: the generalised delta rule with a per-channel decay, and lightning
// attention (linear attention with a constant decay per head; described at its kernel below) with its relatives: retention,
// the state-space scan (a decay per token) and gated linear attention (a decay per token and key channel).
//
// Per head, with a state S [dim x dim] (key channel i, value column j) kept in fp32 per sequence slot:
//     u   = k / sqrt(sum(k^2) + key_eps)
//     S  <- diag(w) S - (a * u) (u^T S) + k v^T          (both first terms read the old S)
//     o   = S^T r
// Everything that enters the recurrence besides the projections themselves is fp32: the decay w, the removal rate a,
// the unit key u, the state and the output.
//
// delta_prep_kernel   (CTA per 8 tokens) : w = exp(-decay_scale * sigmoid(W2 tanh(inner) + w0)) with the W2 product in
//                                         fp32 (a thread owns a channel and walks its W2 row once for the CTA's
//                                         tokens), a = sigmoid(a_pre + a_bias), u; writes one packed fp32 record
//                                         [r | k | w | u | a*u | v] x dp (dp = dim rounded up to 4) per (token, head),
//                                         so that the recurrence streams ONE contiguous block per token and head.
// delta_rule_kernel   (CTA per (sequence segment, head)): the state lives in registers, a thread owning a quarter of
//                                         one value column; the u^T S and S^T r products are per-thread dot products
//                                         with vectors read from shared memory plus two shuffle steps, so the tokens
//                                         of a segment need no block-wide exchange.  The records of the next
//                                         tokens arrive by cp.async into the other half of a double buffer while
//                                         the current ones are consumed.  The state is loaded from / stored to the
//                                         slot's state once per launch, which makes a prompt portion and a single
//                                         decoded token the same case.
// headnorm_gate_kernel (warp per (token, head)): o / rms(o) per head, times a weight (may be absent), times sigmoid(gate)
//                                         or silu(gate), times a constant, rounded to the model dtype as the output projection's operand.
#include "common.cuh"
#include "tc_common.cuh"

namespace pg {

__device__ __forceinline__ float sigmoid_f(float v) { return 1.f / (1.f + expf(-v)); }

constexpr int PREP_TOK = 8;     // tokens per CTA of the prep kernel
constexpr int REC_VECS = 6;     // r, k, w, u, a*u, v
enum { REC_R = 0, REC_K = 1, REC_W = 2, REC_U = 3, REC_AU = 4, REC_V = 5 };

template <typename T>
__global__ void __launch_bounds__(256)
delta_prep_kernel(float* __restrict__ rec, const T* __restrict__ proj, int ld, int r_col0, int k_col0, int v_col0,
                  int a_col0, int lora_col0, int lora, const T* __restrict__ w2, const T* __restrict__ w0,
                  const T* __restrict__ a_bias, int n_tokens, int heads, int dim, int dp, float decay_scale,
                  float key_eps) {
  extern __shared__ float sm[];           // [PREP_TOK][lora] tanh of the decay's inner projection | [PREP_TOK][heads] sum k^2
  float* lo = sm;
  float* ksq = sm + PREP_TOK * lora;
  pdl_launch_dependents();
  pdl_wait();
  const int t0 = blockIdx.x * PREP_TOK, nt = min(PREP_TOK, n_tokens - t0), nd = heads * dim;
  for (int idx = threadIdx.x; idx < PREP_TOK * lora; idx += blockDim.x) {
    const int tt = idx / lora, j = idx % lora;
    lo[idx] = tt < nt ? tanhf(to_f<T>(proj[(size_t)(t0 + tt) * ld + lora_col0 + j])) : 0.f;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int item = warp; item < nt * heads; item += warps) {
    const int tt = item / heads, h = item % heads;
    const T* kr = proj + (size_t)(t0 + tt) * ld + k_col0 + h * dim;
    float s = 0.f;
    for (int c = lane; c < dim; c += 32) { const float v = to_f<T>(kr[c]); s += v * v; }
    s = warp_sum(s);
    if (lane == 0) ksq[tt * heads + h] = s;
  }
  __syncthreads();
  constexpr int V = Vec<T>::N;
  const bool vec = (lora % V) == 0 && (reinterpret_cast<uintptr_t>(w2) & 15) == 0;
  // blockIdx.y cuts the channels into slices of c_per (a handful of tokens: more CTAs than token groups)
  const int c_per = (nd + gridDim.y - 1) / gridDim.y, c_end = min(nd, (int)(blockIdx.y + 1) * c_per);
  for (int c = blockIdx.y * c_per + threadIdx.x; c < c_end; c += blockDim.x) {
    float z[PREP_TOK];
    const float z0 = to_f<T>(w0[c]);
#pragma unroll
    for (int tt = 0; tt < PREP_TOK; ++tt) z[tt] = z0;
    const T* wr = w2 + (size_t)c * lora;
    if (vec) {
      for (int j = 0; j < lora; j += V) {
        float f[V];
        unpack<T>(*reinterpret_cast<const uint4*>(wr + j), f);
#pragma unroll
        for (int tt = 0; tt < PREP_TOK; ++tt)
#pragma unroll
          for (int i = 0; i < V; ++i) z[tt] = fmaf(f[i], lo[tt * lora + j + i], z[tt]);
      }
    } else {
      for (int j = 0; j < lora; ++j) {
        const float f = to_f<T>(wr[j]);
#pragma unroll
        for (int tt = 0; tt < PREP_TOK; ++tt) z[tt] = fmaf(f, lo[tt * lora + j], z[tt]);
      }
    }
    const int h = c / dim, i = c % dim;
    const float ab = a_bias ? to_f<T>(a_bias[c]) : 0.f;
#pragma unroll
    for (int tt = 0; tt < PREP_TOK; ++tt) {
      if (tt >= nt) break;
      const T* row = proj + (size_t)(t0 + tt) * ld;
      const float k = to_f<T>(row[k_col0 + c]);
      const float u = k / sqrtf(ksq[tt * heads + h] + key_eps);
      float* o = rec + (((size_t)(t0 + tt) * heads + h) * REC_VECS) * dp + i;
      o[REC_R * dp] = to_f<T>(row[r_col0 + c]);
      o[REC_K * dp] = k;
      o[REC_W * dp] = expf(-decay_scale * sigmoid_f(z[tt]));
      o[REC_U * dp] = u;
      o[REC_AU * dp] = sigmoid_f(to_f<T>(row[a_col0 + c]) + ab) * u;
      o[REC_V * dp] = to_f<T>(row[v_col0 + c]);
    }
  }
  // the padding columns of every record are zero, so the recurrence can run whole 4-wide groups
  const int pad = dp - dim;
  if (pad && blockIdx.y == 0)
    for (int idx = threadIdx.x; idx < nt * heads * REC_VECS * pad; idx += blockDim.x) {
      const int i = dim + idx % pad, which = idx / pad;
      rec[((size_t)t0 * heads * REC_VECS + which) * dp + i] = 0.f;
    }
}

// segs: [n_segs][3] = {state slot, first token row, tokens}; the tokens of a segment are consecutive rows of one
// sequence in position order.  A segment with 0 tokens is skipped (the list is padded to a fixed length so that a
// captured launch stays valid).  Shared memory: two buffers of CH records.
template <int DMAX, int CH>
__global__ void __launch_bounds__(DMAX * 4)
delta_rule_kernel(float* __restrict__ out, float* __restrict__ state, const float* __restrict__ rec,
                  const int32_t* __restrict__ segs, int heads, int dim, int dp) {
  // thread = (value column j, row group rg): of column j it keeps the rows 4 (m RG + rg) + e (m < NG, e < 4) in
  // registers, i.e. every RG-th group of four rows, so that the four row groups of a column (adjacent lanes) read four
  // consecutive 16-byte pieces of a vector (no bank conflict) and the two column sums of a token are two shuffle
  // steps each.  Vectors sit in shared memory with stride DMAX and zeros behind dim: no bound checks in the token loop.
  constexpr int RG = 4, NG = DMAX / (4 * RG);
  extern __shared__ __align__(16) float sh[];       // [2][CH][REC_VECS][DMAX]
  pdl_launch_dependents();
  pdl_wait();
  const int32_t* sg = segs + 3 * (size_t)blockIdx.x;
  const int slot = sg[0], row0 = sg[1], n = sg[2];
  if (n <= 0) return;
  const int h = blockIdx.y, j = blockIdx.z * (blockDim.x / RG) + threadIdx.x / RG, rg = threadIdx.x % RG, nd = heads * dim;
  const bool live = j < dim;
  constexpr int RSZ = REC_VECS * DMAX;              // floats of one record in shared memory
  if (dp < DMAX)
    for (int idx = threadIdx.x; idx < 2 * CH * RSZ; idx += blockDim.x)
      if (idx % DMAX >= dp) sh[idx] = 0.f;
  float S[NG * 4];
  float* st = state + ((size_t)slot * heads + h) * dim * dim;
#pragma unroll
  for (int m = 0; m < NG; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 4 * (m * RG + rg) + e;
      S[m * 4 + e] = (live && i < dim) ? st[(size_t)i * dim + j] : 0.f;
    }
  const int vp = dp / 4, pieces = REC_VECS * vp;    // 16-byte pieces of one vector / one record
  auto fetch = [&](int t0, int buf) {               // records of tokens [t0, t0 + CH) of this head -> buffer buf
    const int nt = min(CH, n - t0);
    for (int idx = threadIdx.x; idx < nt * pieces; idx += blockDim.x) {
      const int tt = idx / pieces, rem = idx % pieces, v = rem / vp, pc = rem % vp;
      cp_async16(sh + ((size_t)buf * CH + tt) * RSZ + v * DMAX + pc * 4,
                 rec + (((size_t)row0 + t0 + tt) * heads + h) * (size_t)(REC_VECS * dp) + v * dp + pc * 4);
    }
    cp_async_commit();
  };
  fetch(0, 0);
  int buf = 0;
  for (int t0 = 0; t0 < n; t0 += CH, buf ^= 1) {
    const int nt = min(CH, n - t0);
    if (t0 + CH < n) { fetch(t0 + CH, buf ^ 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    __syncthreads();
#pragma unroll 2
    for (int tt = 0; tt < nt; ++tt) {
      const float* r = sh + ((size_t)buf * CH + tt) * RSZ + 4 * rg;
      const float vj = r[REC_V * DMAX + j - 4 * rg];
      float4 u4[NG], w4[NG], a4[NG], k4[NG], r4[NG];
#pragma unroll
      for (int m = 0; m < NG; ++m) {
        u4[m] = *reinterpret_cast<const float4*>(r + REC_U * DMAX + 16 * m);
        w4[m] = *reinterpret_cast<const float4*>(r + REC_W * DMAX + 16 * m);
        a4[m] = *reinterpret_cast<const float4*>(r + REC_AU * DMAX + 16 * m);
        k4[m] = *reinterpret_cast<const float4*>(r + REC_K * DMAX + 16 * m);
        r4[m] = *reinterpret_cast<const float4*>(r + REC_R * DMAX + 16 * m);
      }
      float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;            // this thread's part of u^T S for column j
#pragma unroll
      for (int m = 0; m < NG; ++m) {
        d0 = fmaf(u4[m].x, S[4 * m], d0); d1 = fmaf(u4[m].y, S[4 * m + 1], d1);
        d2 = fmaf(u4[m].z, S[4 * m + 2], d2); d3 = fmaf(u4[m].w, S[4 * m + 3], d3);
      }
      float us = (d0 + d1) + (d2 + d3);
      us += __shfl_xor_sync(0xffffffffu, us, 1);
      us += __shfl_xor_sync(0xffffffffu, us, 2);
      float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
      for (int m = 0; m < NG; ++m) {
        S[4 * m] = fmaf(k4[m].x, vj, fmaf(-a4[m].x, us, w4[m].x * S[4 * m]));
        S[4 * m + 1] = fmaf(k4[m].y, vj, fmaf(-a4[m].y, us, w4[m].y * S[4 * m + 1]));
        S[4 * m + 2] = fmaf(k4[m].z, vj, fmaf(-a4[m].z, us, w4[m].z * S[4 * m + 2]));
        S[4 * m + 3] = fmaf(k4[m].w, vj, fmaf(-a4[m].w, us, w4[m].w * S[4 * m + 3]));
        o0 = fmaf(r4[m].x, S[4 * m], o0); o1 = fmaf(r4[m].y, S[4 * m + 1], o1);
        o2 = fmaf(r4[m].z, S[4 * m + 2], o2); o3 = fmaf(r4[m].w, S[4 * m + 3], o3);
      }
      float o = (o0 + o1) + (o2 + o3);
      o += __shfl_xor_sync(0xffffffffu, o, 1);
      o += __shfl_xor_sync(0xffffffffu, o, 2);
      if (live && rg == 0) out[((size_t)row0 + t0 + tt) * nd + h * dim + j] = o;
    }
    __syncthreads();                                // every thread is done with this buffer before it is refilled
  }
  if (live) {
#pragma unroll
    for (int m = 0; m < NG; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 4 * (m * RG + rg) + e;
        if (i < dim) st[(size_t)i * dim + j] = S[m * 4 + e];
      }
  }
}

template <typename T>
__global__ void headnorm_gate_kernel(T* __restrict__ out, int ld_out, const float* __restrict__ o, const T* __restrict__ w,
                                     const T* __restrict__ gate, int ld_gate, int n_tokens, int heads, int dim, float eps,
                                     float out_scale, int pairs, int gate_silu) {
  pdl_launch_dependents();
  pdl_wait();
  const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (item >= (long long)n_tokens * heads) return;
  const int t = (int)(item / heads), h = (int)(item % heads);
  const float* orow = o + ((size_t)t * heads + h) * dim;
  auto gate_f = [&](float z) { return gate_silu ? z * sigmoid_f(z) : sigmoid_f(z); };
  float ss = 0.f;
  if (pairs) {                                     // two columns per lane and access (even sizes, aligned rows)
    for (int c = 2 * lane; c < dim; c += 64) { const float2 v = *reinterpret_cast<const float2*>(orow + c); ss += v.x * v.x + v.y * v.y; }
    ss = warp_sum(ss);
    const float inv = out_scale / sqrtf(ss / (float)dim + eps);
    for (int c = 2 * lane; c < dim; c += 64) {
      const float2 v = *reinterpret_cast<const float2*>(orow + c);
      float a = v.x * inv, b = v.y * inv;
      if (w) { a *= to_f<T>(w[h * dim + c]); b *= to_f<T>(w[h * dim + c + 1]); }
      if (gate) {
        const T* gp = gate + (size_t)t * ld_gate + h * dim + c;
        a *= gate_f(to_f<T>(gp[0])); b *= gate_f(to_f<T>(gp[1]));
      }
      T* op = out + (size_t)t * ld_out + h * dim + c;
      if constexpr (sizeof(T) == 2) {
        T two[2] = {from_f<T>(a), from_f<T>(b)};
        *reinterpret_cast<uint32_t*>(op) = *reinterpret_cast<const uint32_t*>(two);
      } else {
        op[0] = from_f<T>(a); op[1] = from_f<T>(b);
      }
    }
    return;
  }
  for (int c = lane; c < dim; c += 32) ss += orow[c] * orow[c];
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / (float)dim + eps);
  for (int c = lane; c < dim; c += 32) {
    float v = orow[c] * inv;
    if (w) v *= to_f<T>(w[h * dim + c]);
    if (gate) v *= gate_f(to_f<T>(gate[(size_t)t * ld_gate + h * dim + c]));
    out[(size_t)t * ld_out + h * dim + c] = from_f<T>(v * out_scale);
  }
}

// ------------------------------------------------------------------ lightning attention: linear attention with a constant decay per head
// Per head, with a state S [dim x vdim] (key channel i, value column j) kept in fp32 per sequence slot:
//     q = silu(q_pre), k = silu(k_pre), v = silu(v_pre)          (pre-activations: the fused projection, model dtype)
//     S <- decay_h S + k v^T,        o = S^T q
// lightning_prep_kernel  (elementwise)  the activations in fp32, one packed record [q | k | v] per (token, head) with
//                                       q, k padded to dp = dim rounded up to 4 floats and v to vp likewise (zeros).
// lightning_kernel       (CTA per (sequence segment, head, slice of VT value columns)): a step is four tokens.  With S the state
//                                       before them, E_i the product of the decays up to token i, G_j of those behind token j:
//                                           o_i = (E_i q_i)^T S + sum over j <= i of (q_i . (decays between them) k_j) v_j
//                                           S  <- E_3 S + sum over j of (G_j k_j) v_j^T
//                                       which is nine multiply-adds per state element and step for twelve, and no token of a
//                                       step waits for the one before.  Decays are only multiplied, never divided by, so any
//                                       value keeps its meaning; a token reads nothing of a later one, infinities neither.  (A
//                                       query times a key is taken before the value: where that overflows, or a query is
//                                       infinite, the token's outputs are not finite, NaN where token by token gave infinity.)
//                                       Two warps copy the records (cp.async, several steps ahead), scale q and k and take
//                                       the ten products of a step; up to four hold the state, RG lanes sharing one, two or
//                                       four value columns, a thread rows 4 (m RG + rg) + e of them.  The arithmetic runs on
//                                       pairs of rows (fma.rn.f32x2; 2.4 cycles an SM quarter, 3 from a single warp).
//                                       Bound by those and by the shared-memory reads of q and k: of a step's 1480 cycles
//                                       (64 columns of 128 rows) 890 issue and about 700 multiply.
//                                       4 x 2048 tokens, 16 heads of 128: token by token with the copies in every warp 620
//                                       us, this 375; one sequence of 512 tokens 105 and 62, 8 heads of it 150 and 49; 128 single
//                                       tokens 96 and 86.  A wait that runs out leaves NaN in state and outputs and sets the flag.
//                                       The state is read from and written back to the slot once per launch, which
//                                       makes a prompt portion and a single decoded token the same case; where a sequence
//                                       is cut decides which tokens share a step, and with it the last bits.
template <typename T>
__global__ void lightning_prep_kernel(float* __restrict__ rec, const T* __restrict__ proj, int ld, int q_col0, int k_col0,
                                      int v_col0, long long n_tokens, int heads, int dim, int vdim, int dp, int vp) {
  pdl_launch_dependents();
  pdl_wait();
  const int rs = 2 * dp + vp;                       // floats of one record
  // blockIdx.x: token; the CTA's threads walk the token's heads x record columns
  const long long t = blockIdx.x;
  const T* row = proj + t * ld;
  float* out = rec + t * heads * rs;
  for (int i = threadIdx.x; i < heads * rs; i += blockDim.x) {
    const int h = i / rs, c = i - h * rs;
    int col = -1;
    if (c < dp) { if (c < dim) col = q_col0 + h * dim + c; }
    else if (c < 2 * dp) { if (c - dp < dim) col = k_col0 + h * dim + c - dp; }
    else if (c - 2 * dp < vdim) col = v_col0 + h * vdim + c - 2 * dp;
    float a = 0.f;
    if (col >= 0) {
      a = to_f<T>(row[col]);
      a = a * sigmoid_f(a);
    }
    out[i] = a;
  }
}

// The same with 16-byte loads, for head sizes and rows that are whole vectors: 8 records' columns per thread and step
// (8192 tokens of 16 heads of 128: an element per thread 156 us, this 56 us; 302 MB move).
template <typename T>
__global__ void __launch_bounds__(256)
lightning_prep_vec_kernel(float* __restrict__ rec, const T* __restrict__ proj, int ld, int q_col0, int k_col0, int v_col0,
                          int heads, int dim, int vdim) {
  constexpr int V = Vec<T>::N;
  pdl_launch_dependents();
  pdl_wait();
  const int rs = 2 * dim + vdim, per_head = rs / V;
  const T* row = proj + (size_t)blockIdx.x * ld;
  float* out = rec + (size_t)blockIdx.x * heads * rs;
  for (int i = threadIdx.x; i < heads * per_head; i += blockDim.x) {
    const int h = i / per_head, c = (i - h * per_head) * V;
    const int col = c < dim ? q_col0 + h * dim + c : (c < 2 * dim ? k_col0 + h * dim + c - dim : v_col0 + h * vdim + c - 2 * dim);
    float f[V];
    unpack<T>(ldg_cached(row + col), f);
#pragma unroll
    for (int k = 0; k < V; ++k) f[k] = f[k] * sigmoid_f(f[k]);
    float4* dst = reinterpret_cast<float4*>(out + (size_t)h * rs + c);
#pragma unroll
    for (int k = 0; k < V; k += 4) dst[k / 4] = make_float4(f[k], f[k + 1], f[k + 2], f[k + 3]);
  }
}

// Gated linear attention runs on the same recurrence with a decay per key channel: a = sigmoid(z)^(1/tau), z = W2 inner + b2
// with `inner` the decay's low-rank projection.  The W2 product, the logarithm and the exponential are fp32.  A CTA takes
// PREP_TOK tokens; a thread owns a key channel and walks its W2 row once for all of them.
template <typename T>
__global__ void __launch_bounds__(256)
gla_prep_kernel(float* __restrict__ rec, const T* __restrict__ proj, int ld, int q_col0, int k_col0, int v_col0, int a_col0,
                int rank, const T* __restrict__ w2, const T* __restrict__ b2, float q_scale, float inv_tau, int n_tokens,
                int heads, int dim, int vdim, int dp, int vp) {
  extern __shared__ float lo[];                     // [PREP_TOK][rank]
  pdl_launch_dependents();
  pdl_wait();
  const int t0 = blockIdx.x * PREP_TOK, nt = min(PREP_TOK, n_tokens - t0), rs = 3 * dp + vp;
  for (int idx = threadIdx.x; idx < PREP_TOK * rank; idx += blockDim.x) {
    const int tt = idx / rank, j = idx - tt * rank;
    lo[idx] = tt < nt ? to_f<T>(proj[(size_t)(t0 + tt) * ld + a_col0 + j]) : 0.f;
  }
  __syncthreads();
  constexpr int V = Vec<T>::N;
  const bool vec = (rank % V) == 0 && (reinterpret_cast<uintptr_t>(w2) & 15) == 0;
  // blockIdx.y cuts the columns into slices (a handful of tokens: more CTAs than token groups)
  const int n_key = heads * dp, k_per = (n_key + gridDim.y - 1) / gridDim.y, k_end = min(n_key, (int)(blockIdx.y + 1) * k_per);
  for (int c = blockIdx.y * k_per + threadIdx.x; c < k_end; c += blockDim.x) {
    const int h = c / dp, i = c - h * dp, ch = h * dim + i;
    float z[PREP_TOK];
    const bool in = i < dim;                        // the padding channels of a record are zero
    const float z0 = in ? to_f<T>(b2[ch]) : 0.f;
#pragma unroll
    for (int tt = 0; tt < PREP_TOK; ++tt) z[tt] = z0;
    if (in) {
      const T* wr = w2 + (size_t)ch * rank;
      if (vec) {
        for (int j = 0; j < rank; j += V) {
          float f[V];
          unpack<T>(*reinterpret_cast<const uint4*>(wr + j), f);
#pragma unroll
          for (int tt = 0; tt < PREP_TOK; ++tt)
#pragma unroll
            for (int k = 0; k < V; ++k) z[tt] = fmaf(f[k], lo[tt * rank + j + k], z[tt]);
        }
      } else {
        for (int j = 0; j < rank; ++j) {
          const float f = to_f<T>(wr[j]);
#pragma unroll
          for (int tt = 0; tt < PREP_TOK; ++tt) z[tt] = fmaf(f, lo[tt * rank + j], z[tt]);
        }
      }
    }
#pragma unroll
    for (int tt = 0; tt < PREP_TOK; ++tt) {
      if (tt >= nt) break;
      const T* row = proj + (size_t)(t0 + tt) * ld;
      float* o = rec + ((size_t)(t0 + tt) * heads + h) * rs + i;
      o[0] = in ? to_f<T>(row[q_col0 + ch]) * q_scale : 0.f;
      o[dp] = in ? to_f<T>(row[k_col0 + ch]) : 0.f;
      o[2 * dp] = in ? expf((fminf(z[tt], 0.f) - log1pf(expf(-fabsf(z[tt])))) * inv_tau) : 0.f;
    }
  }
  const int n_val = heads * vp, v_per = (n_val + gridDim.y - 1) / gridDim.y, v_end = min(n_val, (int)(blockIdx.y + 1) * v_per);
  for (int c = blockIdx.y * v_per + threadIdx.x; c < v_end; c += blockDim.x) {
    const int h = c / vp, i = c - h * vp;
    for (int tt = 0; tt < nt; ++tt)
      rec[((size_t)(t0 + tt) * heads + h) * rs + 3 * dp + i] =
          i < vdim ? to_f<T>(proj[(size_t)(t0 + tt) * ld + v_col0 + h * vdim + i]) : 0.f;
  }
}

// Retention (linear attention with rotary positions in place of activations) runs on the same recurrence: its records
// are written by retention_prep_kernel below.  The first rot_dims columns of every q and k head are turned in pairs
// (i, i + rot_dims / 2), or (2i, 2i + 1) when interleaved, by position * freq[i]; k is multiplied by k_scale after the
// rotation; v passes.  freq holds (high, low) float pairs (rotary_sincos).  One CTA per token: the token's sines and cosines
// once into shared memory (the heads share them), then records four columns at a time.
template <typename T>
__global__ void retention_prep_kernel(float* __restrict__ rec, const T* __restrict__ proj, int ld, int q_col0, int k_col0,
                                      int v_col0, const float2* __restrict__ freq, int rot_dims, int interleaved, float k_scale,
                                      const int32_t* __restrict__ tok_pos, int heads, int dim, int vdim, int dp, int vp) {
  extern __shared__ float2 cs[];                    // [rot_dims / 2] (cos, sin)
  pdl_launch_dependents();
  pdl_wait();
  const long long t = blockIdx.x;
  const int half = rot_dims >> 1, rs = 2 * dp + vp, rs4 = rs / 4;
  const float p = (float)tok_pos[t];
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    const float2 f = freq[i];
    float s, c;
    rotary_sincos(p, f.x, f.y, &s, &c);
    cs[i] = make_float2(c, s);
  }
  __syncthreads();
  const T* row = proj + t * ld;
  float* out = rec + t * heads * rs;
  auto rotated = [&](const T* head, int c) -> float {          // column c of a q or k head
    const float u = to_f<T>(head[c]);
    if (c >= rot_dims) return u;
    const bool first = interleaved ? !(c & 1) : c < half;
    const int pair = interleaved ? c >> 1 : (first ? c : c - half);
    const float w = to_f<T>(head[interleaved ? c ^ 1 : (first ? c + half : c - half)]);
    const float2 e = cs[pair];
    return first ? u * e.x - w * e.y : u * e.x + w * e.y;
  };
  // pairs of halves with everything in whole groups of four: 8- or 16-byte loads
  const bool quad = !interleaved && half % 4 == 0 && dim % 4 == 0 && vdim % 4 == 0 && ld % 4 == 0 && q_col0 % 4 == 0 &&
                    k_col0 % 4 == 0 && v_col0 % 4 == 0 && (reinterpret_cast<uintptr_t>(proj) & 15) == 0;
  auto ld4 = [&](const T* q, float* f) {
    if constexpr (sizeof(T) == 4) {
      const float4 v = *reinterpret_cast<const float4*>(q);
      f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    } else {
      const uint2 v = *reinterpret_cast<const uint2*>(q);
      const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int k = 0; k < 4; ++k) f[k] = to_f<T>(e[k]);
    }
  };
  for (int i = threadIdx.x; i < heads * rs4; i += blockDim.x) {
    const int h = i / rs4, c0 = (i - h * rs4) * 4;
    float o[4] = {0.f, 0.f, 0.f, 0.f};
    if (c0 >= 2 * dp) {
      const int c = c0 - 2 * dp;
      const T* head = row + v_col0 + h * vdim;
      if (quad) { ld4(head + c, o); }
      else {
#pragma unroll
        for (int k = 0; k < 4; ++k) if (c + k < vdim) o[k] = to_f<T>(head[c + k]);
      }
    } else {
      const bool is_k = c0 >= dp;
      const int c = is_k ? c0 - dp : c0;
      const T* head = row + (is_k ? k_col0 : q_col0) + h * dim;
      const float sc = is_k ? k_scale : 1.f;
      if (quad) {
        float u[4];
        ld4(head + c, u);
        if (c < rot_dims) {
          const bool first = c < half;
          const int pair = first ? c : c - half;
          float w[4];
          ld4(head + (first ? c + half : c - half), w);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 e = cs[pair + k];
            u[k] = first ? u[k] * e.x - w[k] * e.y : u[k] * e.x + w[k] * e.y;
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = u[k] * sc;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) if (c + k < dim) o[k] = rotated(head, c + k) * sc;
      }
    }
    *reinterpret_cast<float4*>(out + (size_t)h * rs + c0) = make_float4(o[0], o[1], o[2], o[3]);
  }
}

//                                       DK (where the decay comes from): DECAY_HEAD decay[h]; DECAY_TOKEN: the record carries
//                                       four more floats [decay, 0, 0, 0] after the values; DECAY_CHANNEL: a vector of dp
//                                       decays between key and values, one per key channel (gated linear attention);
//                                       skip (may be NULL): skip[h] * v is added to the output (the state-space
//                                       mixer's direct term, with v its unscaled input).
enum { DECAY_HEAD = 0, DECAY_TOKEN = 1, DECAY_CHANNEL = 2 };

constexpr int SCAN_TB = 4, SCAN_AUX = 2;                  // tokens per step, warps that prepare steps
constexpr int SCAN_SIDE = 20;                             // floats beside a step: weights [4][4], the step's whole decay

// A thread's part of a state: COLS value columns from j on, rows 4 (m RG + rg) + e (m < NG, e < 4) of them, in pairs of rows.
template <int RG, int NG, int COLS>
struct ScanState {
  f32x2 S[COLS][NG * 2];
  static __device__ __forceinline__ void load_row(float* x, const float* p) {
    if constexpr (COLS == 4) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(p);
    else if constexpr (COLS == 2) *reinterpret_cast<float2*>(x) = *reinterpret_cast<const float2*>(p);
    else x[0] = p[0];
  }
  static __device__ __forceinline__ void store_row(float* p, const float* x) {
    if constexpr (COLS == 4) *reinterpret_cast<float4*>(p) = *reinterpret_cast<const float4*>(x);
    else if constexpr (COLS == 2) *reinterpret_cast<float2*>(p) = *reinterpret_cast<const float2*>(x);
    else p[0] = x[0];
  }
  // wide: whole aligned groups of columns; with all rows there too, nothing is asked per row (a branch for each delays the next
  // one's load)
  __device__ __forceinline__ void load(const float* st, int dim, int vdim, int j, int rg, bool wide) {
    if (wide && dim == 4 * NG * RG) {
      float x[NG * 4][COLS];
#pragma unroll
      for (int m = 0; m < NG; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) load_row(x[m * 4 + e], st + (size_t)(4 * (m * RG + rg) + e) * vdim + j);
#pragma unroll
      for (int y = 0; y < NG * 2; ++y)
#pragma unroll
        for (int c = 0; c < COLS; ++c) S[c][y] = pair_of(x[2 * y][c], x[2 * y + 1][c]);
      return;
    }
#pragma unroll
    for (int m = 0; m < NG; ++m)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          const int i = 4 * (m * RG + rg) + e;
          const float* p = st + (size_t)i * vdim + j + c;
          const bool col = j + c < vdim;
          S[c][m * 2 + e / 2] = pair_of(col && i < dim ? p[0] : 0.f, col && i + 1 < dim ? p[vdim] : 0.f);
        }
  }
  __device__ __forceinline__ void store(float* st, int dim, int vdim, int j, int rg, bool wide) const {
    const bool whole = wide && dim == 4 * NG * RG;
#pragma unroll
    for (int m = 0; m < NG; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 4 * (m * RG + rg) + e;
        float* p = st + (size_t)i * vdim + j;
        float x[COLS];
#pragma unroll
        for (int c = 0; c < COLS; ++c) { const float2 y = halves_of(S[c][m * 2 + e / 2]); x[c] = e & 1 ? y.y : y.x; }
        if (whole) store_row(p, x);
        else
#pragma unroll
          for (int c = 0; c < COLS; ++c) if (i < dim && j + c < vdim) p[c] = x[c];
      }
  }
  // A few tokens, one after the other, from the records themselves (r: the first one's, tok floats apart).
  template <int DK>
  __device__ __forceinline__ void tokens(float* out, const float* r, size_t tok, int n, const float* decay, int h, int heads, float skip_h,
                                         int vdim, int dp, int vp, int j, int rg) {
    constexpr bool TD = DK == DECAY_TOKEN, CD = DK == DECAY_CHANNEL;
    constexpr int NV = CD ? 3 : 2;
    for (int t = 0; t < n; ++t, r += tok, out += (size_t)heads * vdim) {
      const float lam = TD ? __ldg(r + NV * dp + vp) : (CD ? 1.f : decay[h]);
      float v[COLS];
      f32x2 v2[COLS], o[COLS];
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        v[c] = j + c < vp ? __ldg(r + NV * dp + j + c) : 0.f;
        v2[c] = pair_of(v[c], v[c]);
        o[c] = 0ull;
      }
#pragma unroll
      for (int m = 0; m < NG; ++m) {
        const int i = 4 * (m * RG + rg);
        const ulonglong2 z = make_ulonglong2(0ull, 0ull);
        const ulonglong2 q4 = i < dp ? __ldg(reinterpret_cast<const ulonglong2*>(r + i)) : z;
        const ulonglong2 k4 = i < dp ? __ldg(reinterpret_cast<const ulonglong2*>(r + dp + i)) : z;
        ulonglong2 a4 = make_ulonglong2(pair_of(lam, lam), pair_of(lam, lam));
        if (CD) a4 = i < dp ? __ldg(reinterpret_cast<const ulonglong2*>(r + 2 * dp + i)) : z;
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          S[c][2 * m] = fma2(k4.x, v2[c], mul2(a4.x, S[c][2 * m]));
          S[c][2 * m + 1] = fma2(k4.y, v2[c], mul2(a4.y, S[c][2 * m + 1]));
          o[c] = fma2(q4.x, S[c][2 * m], o[c]);
          o[c] = fma2(q4.y, S[c][2 * m + 1], o[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        const float2 x = halves_of(o[c]);
        float y = x.x + x.y;
#pragma unroll
        for (int w = RG / 2; w >= 1; w >>= 1) y += __shfl_xor_sync(0xffffffffu, y, w);
        if (rg == c % RG && j + c < vdim) out[(size_t)h * vdim + j + c] = fmaf(skip_h, v[c], y);
      }
    }
  }
};

// The wait of a whole warp: a phase that is over costs one try and a vote (the loop with its limit: 200 cycles).
__device__ __forceinline__ bool scan_wait(uint32_t bar, uint32_t parity, volatile int* fail) {
  if (__all_sync(0xffffffffu, tc::mbar_try_wait(bar, parity))) return true;
  return tc::mbar_wait_lim_warp(bar, parity, fail);
}

// p = a b with its rounding error (exact while p is a normal number)
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& err) { p = a * b; err = fmaf(a, b, -p); }

// steps in shared memory: those of a warp are requested this many rounds ahead, less one
template <int DMAX, int DK> constexpr int SCAN_AHEAD = DMAX <= 128 ? 4 : (DK == DECAY_CHANNEL ? 2 : 3);

constexpr int scan_lanes(int dmax) { return dmax == 32 ? 4 : (dmax <= 128 ? 8 : 16); }   // lanes that share value columns

template <int DMAX, int DK, int COLS>           // COLS: value columns per thread, 1, 2 or 4
__global__ void __launch_bounds__((4 + SCAN_AUX) * 32, 2)
lightning_kernel(float* __restrict__ out, float* __restrict__ state, const float* __restrict__ rec,
                 const float* __restrict__ decay, const float* __restrict__ skip, const int32_t* __restrict__ segs,
                 int heads, int dim, int vdim, int dp, int vp, int vec, int no_wait, int* __restrict__ err_flag) {
  constexpr int AHEAD = SCAN_AHEAD<DMAX, DK>, SCAN_RING = AHEAD * SCAN_AUX;
  constexpr int RG = scan_lanes(DMAX), NG = DMAX / (4 * RG), TB = SCAN_TB;   // RG lanes share COLS value columns, NG groups of four rows each
  extern __shared__ __align__(16) float sh[];         // [ring][TB][q DMAX | k DMAX | (decays DMAX) | v VT | (decay)] | [ring][side]
  __shared__ __align__(8) uint64_t bars[2 * SCAN_RING];
  __shared__ int fail;
  pdl_launch_dependents();
  pdl_wait();
  const int32_t* sg = segs + 3 * (size_t)blockIdx.x;
  const int slot = sg[0], row0 = sg[1], n = sg[2];
  if (n <= 0) return;
  constexpr bool TD = DK == DECAY_TOKEN, CD = DK == DECAY_CHANNEL;
  constexpr int XP = TD ? 4 : 0, NV = CD ? 3 : 2;     // NV: vectors of key width in a record
  const int nw = (int)(blockDim.x >> 5) - SCAN_AUX, VT = COLS * (32 / RG) * nw;
  const int RSZ = NV * DMAX + VT + XP, rs = NV * dp + vp + XP, steps = (n + TB - 1) / TB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.y, j0 = blockIdx.z * VT;
  const float* head_rec = rec + ((size_t)row0 * heads + h) * (size_t)rs;   // token t's record: + t * heads * rs
  const size_t tok_step = (size_t)heads * rs;
  float* side = sh + (size_t)SCAN_RING * TB * RSZ;
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bars);
  auto ready = [&](int s) { return bar0 + 8u * s; };                      // the step is prepared
  auto empty = [&](int s) { return bar0 + 8u * (SCAN_RING + s); };        // every warp has used it
  const bool direct = n < TB;                         // a few tokens: no ring, each state warp reads the records itself
  if (direct) {
    if (warp >= nw) return;
  } else {
    if (threadIdx.x == 0) {
      for (int s = 0; s < SCAN_RING; ++s) { tc::mbar_init(ready(s), 1); tc::mbar_init(empty(s), nw); }
      fail = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
  }

  if (warp >= nw) {
    // ---- a step's records and what it needs besides, by one warp: with E_i the product of the decays up to token i and G_j of
    // those behind token j, q_i <- E_i q_i, k_j <- G_j k_j, and the weight of v_j in token i's output, w_ij = q_i . (the decays
    // between them) k_j.  Tokens behind the segment's last are zeros that decay by 1.  The copies run AHEAD - 1 of this warp's
    // steps ahead (plain loads into registers shared their scoreboards with the shuffles: 3000 cycles a step instead of 600).
    constexpr int F4 = (DMAX / 4 + 31) / 32;
    const float lam_h = DK == DECAY_HEAD ? decay[h] : 1.f;
    // values: 16-byte pieces of the step's tokens, V4 per lane (VT / 4 is a power of two up to 32)
    constexpr int V4 = (COLS * (32 / RG) * 4 + 31) / 32;
    const int v_len = min(VT, vp - j0), v_pieces = VT / 4, v_tok = lane / v_pieces, v_col = 4 * (lane % v_pieces), v_tstep = 32 / v_pieces;
    float carry[CD ? F4 : 1][4];                        // what the roundings of the whole decays have added up to (relative)
#pragma unroll
    for (int f = 0; f < (CD ? F4 : 1); ++f)
#pragma unroll
      for (int e = 0; e < 4; ++e) carry[f][e] = 0.f;
    bool lost = no_wait != 0;                           // the state's warps have stopped
    auto request = [&](int it) {
      // the state's warps have read the slot (in a first round nobody has to)
      if (it >= SCAN_RING && it < steps) lost = !scan_wait(empty(it % SCAN_RING), (it / SCAN_RING - 1) & 1, &fail);
      if (it < steps && !lost) {
        const int s = it % SCAN_RING, nv = min(TB, n - it * TB);
        const float* src = head_rec + (size_t)it * TB * tok_step;
        float* dst = sh + (size_t)s * TB * RSZ;
#pragma unroll
        for (int t = 0; t < TB; ++t) {
          const float* p = src + t * tok_step;
          float* d = dst + t * RSZ;
#pragma unroll
          for (int f = 0; f < F4; ++f) {
            const int c = 4 * (lane + 32 * f);
            const bool have = t < nv && c < dp;
#pragma unroll
            for (int x = 0; x < NV; ++x) if (have) cp_async16(d + x * DMAX + c, p + x * dp + c);
          }
          if (TD && lane == 31 && t < nv) cp_async16(d + NV * DMAX + VT, p + NV * dp + vp);
        }
#pragma unroll
        for (int x = 0; x < V4; ++x)
          if (v_tok + x * v_tstep < nv && v_col < v_len)
            cp_async16(dst + (v_tok + x * v_tstep) * RSZ + NV * DMAX + v_col, src + (v_tok + x * v_tstep) * tok_step + NV * dp + j0 + v_col);
      }
      cp_async_commit();
    };
    const int first = warp - nw;
#pragma unroll 1
    for (int i = 0; i < AHEAD - 1; ++i) request(first + i * SCAN_AUX);
    for (int it = first; it < steps; it += SCAN_AUX) {
      cp_async_wait<AHEAD - 2>();
      __syncwarp();
      if (lost) break;
      const int s = it % SCAN_RING, nv = min(TB, n - it * TB);
      float* base = sh + (size_t)s * TB * RSZ;
      float* sd = side + (size_t)s * SCAN_SIDE;
      float q[F4][TB][4], k[F4][TB][4], a[CD ? F4 : 1][TB][4], lam[TB];
#pragma unroll
      for (int t = 0; t < TB; ++t) {
        lam[t] = t >= nv ? 1.f : (TD ? base[t * RSZ + NV * DMAX + VT] : lam_h);
#pragma unroll
        for (int f = 0; f < F4; ++f) {
          const int c = 4 * (lane + 32 * f);
          const bool have = t < nv && c < dp;
          const float4 z = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
          const float* p = base + t * RSZ + c;
          *reinterpret_cast<float4*>(q[f][t]) = have ? *reinterpret_cast<const float4*>(p) : z;
          *reinterpret_cast<float4*>(k[f][t]) = have ? *reinterpret_cast<const float4*>(p + DMAX) : z;
          if constexpr (CD) *reinterpret_cast<float4*>(a[f][t]) = have ? *reinterpret_cast<const float4*>(p + 2 * DMAX) : one;
        }
        if (t >= nv)
          for (int c = lane; c < VT; c += 32) base[t * RSZ + NV * DMAX + c] = 0.f;
      }
      float w[16];                                      // the weights of token pairs j <= i, at i (i + 1) / 2 + j
#pragma unroll
      for (int x = 0; x < 16; ++x) w[x] = 0.f;
      // The whole decay of a step multiplies the state once per step: rounded the same way every time its error would add up over
      // the steps (a constant decay near 1 above all), so the part that the last roundings lost is put back into the next one.
      auto whole = [&](float p, float err, float& carry) {
        const float fix = fmaf(p, carry, err), d = p + fix;
        carry = p > 1e-30f ? ((p - d) + fix) / p : 0.f;
        return d;
      };
      float E[TB], G[TB], D = 1.f;
      if constexpr (!CD) {
        float p = lam[0], err = 0.f;
        E[0] = p;
#pragma unroll
        for (int i = 1; i < TB; ++i) {
          float x, y;
          two_prod(p, lam[i], x, y);
          err = fmaf(err, lam[i], y);
          p = x;
          E[i] = p + err;
        }
        D = whole(p, err, carry[0][0]);
        G[TB - 1] = 1.f;
        p = 1.f; err = 0.f;
#pragma unroll
        for (int i = TB - 2; i >= 0; --i) {
          float x, y;
          two_prod(p, lam[i + 1], x, y);
          err = fmaf(err, lam[i + 1], y);
          p = x;
          G[i] = p + err;
        }
      }
#pragma unroll
      for (int f = 0; f < F4; ++f) {
        const int c = 4 * (lane + 32 * f);
        if (c >= DMAX) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float p = 1.f, err = 0.f;
#pragma unroll
          for (int i = 0; i < TB; ++i) {
            const float ai = CD ? a[f][i][e] : lam[i];
#pragma unroll
            for (int j = 0; j <= i; ++j) {
              // token j's key decayed up to token i
              if (CD && j < i) k[f][j][e] *= ai;
              w[i * (i + 1) / 2 + j] = fmaf(q[f][i][e], k[f][j][e], w[i * (i + 1) / 2 + j]);
            }
            if constexpr (CD) {
              float x, y;
              two_prod(p, ai, x, y);
              err = fmaf(err, ai, y);
              p = x;
              q[f][i][e] *= p + err;
            } else {
              q[f][i][e] *= E[i];
            }
          }
          if constexpr (CD) {
            a[f][0][e] = whole(p, err, carry[f][e]);
          } else {
#pragma unroll
            for (int j = 0; j < TB - 1; ++j) k[f][j][e] *= G[j];
          }
        }
#pragma unroll
        for (int t = 0; t < TB; ++t) {
          *reinterpret_cast<float4*>(base + t * RSZ + c) = *reinterpret_cast<const float4*>(q[f][t]);
          *reinterpret_cast<float4*>(base + t * RSZ + DMAX + c) = *reinterpret_cast<const float4*>(k[f][t]);
        }
        if constexpr (CD) *reinterpret_cast<float4*>(base + 2 * DMAX + c) = *reinterpret_cast<const float4*>(a[f][0]);
      }
      float between[TB][TB];                            // the decays between two tokens, where one number per token does
      if constexpr (!CD) {
#pragma unroll
        for (int j = 0; j < TB; ++j) {
          between[j][j] = 1.f;
#pragma unroll
          for (int i = j + 1; i < TB; ++i) between[i][j] = between[i - 1][j] * lam[i];
        }
      }
#pragma unroll
      for (int o = 16, m = 8; o >= 2; o >>= 1, m >>= 1) {   // a transposed butterfly: lane L ends up with half of sum L / 2
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int x = 0; x < m; ++x) {
          const float keep = up ? w[x + m] : w[x], send = up ? w[x] : w[x + m];
          w[x] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      w[0] += __shfl_xor_sync(0xffffffffu, w[0], 1);
      // one store for the warp, chosen without branches (a branch per weight cost 2400 cycles a step)
      float mine = lane == 31 ? D : w[0];
      int at = lane == 31 ? 16 : 17;                    // 17: nobody's
#pragma unroll
      for (int i = 0; i < TB; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
          const bool is = lane == 2 * (i * (i + 1) / 2 + j);
          if (!CD && j < i) mine = is ? mine * between[i][j] : mine;
          at = is ? 4 * i + j : at;
        }
      sd[at] = mine;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(ready(s));
      request(it + (AHEAD - 1) * SCAN_AUX);
    }
    // A wait that ran out, here or in a state's warp (which then waited for one of these two): the flag and the outputs show it.
    // These warps tell it: values kept for it in the state's loop cost 6 of 380 us at 4 x 2048 tokens.
    cp_async_wait<0>();
    if (__any_sync(0xffffffffu, lost || *(volatile int*)&fail)) {
      if (lane == 0 && err_flag) *err_flag = 2;
      float* o = out + ((size_t)row0 * heads + h) * vdim + j0;
      for (int t = 0; t < n; ++t, o += (size_t)heads * vdim)
        for (int c = lane; c < min(VT, vdim - j0); c += 32) o[c] = __int_as_float(0x7fffffff);
    }
    return;
  }

  // ---- the state's warps
  const int jl = COLS * (threadIdx.x / RG), j = j0 + jl, rg = threadIdx.x % RG;
  const float skip_h = skip ? skip[h] : 0.f;
  float* st = state + ((size_t)slot * heads + h) * dim * vdim;
  const bool wide = vec && j + COLS <= vdim;
  ScanState<RG, NG, COLS> mine;
  auto& S = mine.S;                                   // [column][pair of rows]
  mine.load(st, dim, vdim, j, rg, wide);
  if (direct) {
    mine.template tokens<DK>(out + (size_t)row0 * heads * vdim, head_rec, tok_step, n, decay, h, heads, skip_h, vdim, dp, vp, j, rg);
    mine.store(st, dim, vdim, j, rg, wide);
    return;
  }
  // A step has SUMS column sums.  A transposed butterfly halves their number with every exchange while there are several: lane rg
  // ends up with the PER sums from rg * PER on, or (more lanes than sums) with sum rg / REP.  Sum x: token x / COLS, column x % COLS.
  constexpr int SUMS = TB * COLS, PER = SUMS >= RG ? SUMS / RG : 1, REP = SUMS >= RG ? 1 : RG / SUMS;
  static_assert(COLS % PER == 0, "the sums of a lane belong to one token");
  const int sum0 = rg * PER / REP, my_t = sum0 / COLS, my_c = sum0 % COLS;
  float* orow = out + ((size_t)row0 + my_t) * heads * vdim + (size_t)h * vdim + j + my_c;
  const size_t ostep = (size_t)TB * heads * vdim;
  const int last = no_wait ? 0 : steps;
  int it = 0;
  for (; it < last; ++it, orow += ostep) {
    const int s = it % SCAN_RING;
    if (!scan_wait(ready(s), (it / SCAN_RING) & 1, &fail)) break;
    const float* r0 = sh + (size_t)s * TB * RSZ;
    const float* sd = side + (size_t)s * SCAN_SIDE;
    // what the step's tokens read from the state before it
    f32x2 o[TB][COLS];
    ulonglong2 x4[2][TB];                             // the next group's rows are requested before this one's are used
    auto rows = [&](int which, int m, ulonglong2 (&x)[TB]) {
#pragma unroll
      for (int t = 0; t < TB; ++t) x[t] = *reinterpret_cast<const ulonglong2*>(r0 + t * RSZ + which * DMAX + 4 * rg + 4 * RG * m);
    };
    rows(0, 0, x4[0]);
#pragma unroll
    for (int m = 0; m < NG; ++m) {
      if (m + 1 < NG) rows(0, m + 1, x4[(m + 1) & 1]);
      else rows(1, 0, x4[NG & 1]);
#pragma unroll
      for (int t = 0; t < TB; ++t)
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          o[t][c] = m ? fma2(x4[m & 1][t].x, S[c][2 * m], o[t][c]) : mul2(x4[0][t].x, S[c][0]);
          o[t][c] = fma2(x4[m & 1][t].y, S[c][2 * m + 1], o[t][c]);
        }
    }
    float c_sum[SUMS];
#pragma unroll
    for (int t = 0; t < TB; ++t)
#pragma unroll
      for (int c = 0; c < COLS; ++c) { const float2 x = halves_of(o[t][c]); c_sum[t * COLS + c] = x.x + x.y; }
#pragma unroll
    for (int w = RG / 2, k = SUMS / 2; w >= 1; w >>= 1, k >>= 1) {   // the order of the additions is that of the lanes
      if (k == 0) {
        c_sum[0] += __shfl_xor_sync(0xffffffffu, c_sum[0], w);
        continue;
      }
      const bool up = (rg & w) != 0;
#pragma unroll
      for (int i = 0; i < k; ++i) {
        const float keep = up ? c_sum[i + k] : c_sum[i], send = up ? c_sum[i] : c_sum[i + k];
        c_sum[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
      }
    }
    // the state behind the step
    f32x2 v[TB][COLS];
#pragma unroll
    for (int t = 0; t < TB; ++t) {
      float x[COLS];
      const float* vs = r0 + t * RSZ + NV * DMAX + jl;
      if constexpr (COLS == 4) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(vs);
      else if constexpr (COLS == 2) *reinterpret_cast<float2*>(x) = *reinterpret_cast<const float2*>(vs);
      else x[0] = vs[0];
#pragma unroll
      for (int c = 0; c < COLS; ++c) v[t][c] = pair_of(x[c], x[c]);
    }
    const float whole = CD ? 1.f : sd[16];
    const f32x2 d2 = pair_of(whole, whole);
#pragma unroll
    for (int m = 0; m < NG; ++m) {
      ulonglong2 a4 = make_ulonglong2(d2, d2);
      if (CD) a4 = *reinterpret_cast<const ulonglong2*>(r0 + 2 * DMAX + 4 * rg + 4 * RG * m);
#pragma unroll
      for (int c = 0; c < COLS; ++c) { S[c][2 * m] = mul2(a4.x, S[c][2 * m]); S[c][2 * m + 1] = mul2(a4.y, S[c][2 * m + 1]); }
      if (m + 1 < NG) rows(1, m + 1, x4[(NG + m + 1) & 1]);
#pragma unroll
      for (int t = 0; t < TB; ++t)
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
          S[c][2 * m] = fma2(x4[(NG + m) & 1][t].x, v[t][c], S[c][2 * m]);
          S[c][2 * m + 1] = fma2(x4[(NG + m) & 1][t].y, v[t][c], S[c][2 * m + 1]);
        }
    }
    // the step's own tokens, up to this lane's one, and the direct term
    {
      const float* vs = r0 + NV * DMAX + jl + my_c;
      const bool writes = rg % REP == 0 && it * TB + my_t < n;
#pragma unroll
      for (int x = 0; x < PER; ++x) {
        float y = c_sum[x];
#pragma unroll
        for (int t = 0; t < TB; ++t) y = t <= my_t ? fmaf(sd[4 * my_t + t], vs[t * RSZ + x], y) : y;
        if (writes && j + my_c + x < vdim) orow[x] = fmaf(skip_h, vs[my_t * RSZ + x], y);
      }
    }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(empty(s));
  }
  if (it < steps) {                                   // a wait ran out: the state shows it, and the warps that prepare steps are told
    const float nan = __int_as_float(0x7fffffff);
    if (lane == 0) *(volatile int*)&fail = 1;
#pragma unroll
    for (int c = 0; c < COLS; ++c)
#pragma unroll
      for (int x = 0; x < NG * 2; ++x) S[c][x] = pair_of(nan, nan);
  }
  mine.store(st, dim, vdim, j, rg, wide);
}

template <int DMAX, int COLS>
static int launch_scan_cols(float* out, float* state, const float* rec, const float* decay, const float* skip, int dk,
                            const int32_t* segs, int n_segs, int heads, int dim, int vdim, int no_wait, int* err, cudaStream_t st) {
  const int dp = (dim + 3) / 4 * 4, vp = (vdim + 3) / 4 * 4;
  // value columns per CTA: those of four warps, of fewer while the CTAs do not fill the SMs or the columns are fewer
  constexpr int WARP_COLS = 32 / scan_lanes(DMAX) * COLS;
  int nw = 4;
  while (nw > 1 && (nw / 2) * WARP_COLS >= 4 && ((nw / 2) * WARP_COLS >= vdim || (long long)n_segs * heads * cdiv(vdim, nw * WARP_COLS) < 100))
    nw /= 2;
  const int vt = nw * WARP_COLS;
  const int ring = SCAN_AUX * (dk == DECAY_CHANNEL ? SCAN_AHEAD<DMAX, DECAY_CHANNEL> : SCAN_AHEAD<DMAX, DECAY_HEAD>);
  const size_t smem = sizeof(float) * ring * (SCAN_TB * ((dk == DECAY_CHANNEL ? 3 : 2) * DMAX + vt + (dk == DECAY_TOKEN ? 4 : 0)) + SCAN_SIDE);
  // An ordinary launch, not a programmatic dependent one: CTAs that become resident while the preceding kernel still
  // fills the machine are placed on the few SMs with room, and a recurrence of a few hundred long-lived CTAs then runs
  // on a fraction of the GPU (measured at 4 x 2048 tokens, 8 heads of 128: 2.06 ms against 0.88 ms).
  auto kern = dk == DECAY_CHANNEL ? lightning_kernel<DMAX, DECAY_CHANNEL, COLS>
                                  : (dk == DECAY_TOKEN ? lightning_kernel<DMAX, DECAY_TOKEN, COLS> : lightning_kernel<DMAX, DECAY_HEAD, COLS>);
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    set_error("lightning: cannot reserve %zu B of shared memory", smem);
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  const int vec = COLS == 1 || (vdim % COLS == 0 && (uintptr_t)state % 16 == 0);
  kern<<<dim3(n_segs, heads, cdiv(vdim, vt)), dim3((nw + SCAN_AUX) * 32), smem, st>>>(out, state, rec, decay, skip, segs, heads, dim, vdim,
                                                                                        dp, vp, vec, no_wait, err);
  return check_launch("lightning");
}

template <int DMAX>
static int launch_scan(float* out, float* state, const float* rec, const float* decay, const float* skip, int dk,
                       const int32_t* segs, int n_segs, int heads, int dim, int vdim, int no_wait, int* err, cudaStream_t st) {
  // Value columns per thread: more of them share a token's reads of q and k, but are fewer warps.  By the warps of the one-column
  // form; 512 tokens, us with one, two and four: 128 channels, 1024 columns 49, 60, 92; 4096 98, 76, 92; 8192 193, 113, 107;
  // 64 channels, 4096 72, 58, 55; 256 channels (twice the lanes a column), 2048 113, 84, 91; 4096 220, 126, 117.
  const long long warps = (long long)n_segs * heads * vdim * scan_lanes(DMAX) / 32;
  if (warps >= 1536) return launch_scan_cols<DMAX, 4>(out, state, rec, decay, skip, dk, segs, n_segs, heads, dim, vdim, no_wait, err, st);
  if (warps >= 768) return launch_scan_cols<DMAX, 2>(out, state, rec, decay, skip, dk, segs, n_segs, heads, dim, vdim, no_wait, err, st);
  return launch_scan_cols<DMAX, 1>(out, state, rec, decay, skip, dk, segs, n_segs, heads, dim, vdim, no_wait, err, st);
}

template <int DMAX, int CH>
static int launch_delta(float* out, float* state, const float* rec, const int32_t* segs, int n_segs, int heads, int dim,
                        cudaStream_t st) {
  const int dp = (dim + 3) / 4 * 4;
  const size_t smem = sizeof(float) * 2 * CH * REC_VECS * DMAX;
  // few (segment, head) pairs: the value columns of a head are cut over `cut` CTAs (each fetches the head's records)
  static const int cut_env = env_int("PG_DELTA_COLUMN_CUT", 0);
  int cut = 1;
  if (DMAX >= 16 && (long long)n_segs * heads * 2 <= 160) cut = 2;   // measured: 0.95 -> 0.68 ms at 64 pairs, slower from 128 on
  if (cut_env > 0 && DMAX / cut_env >= 8) cut = cut_env;
  return launch_pdl("delta_rule", delta_rule_kernel<DMAX, CH>, dim3(n_segs, heads, cut), dim3(DMAX * 4 / cut), smem, st, out, state,
                    rec, segs, heads, dim, dp);
}

}  // namespace pg

using namespace pg;

extern "C" long long pg_delta_record_floats(int n_tokens, int heads, int dim) {
  return (long long)n_tokens * heads * REC_VECS * ((dim + 3) / 4 * 4);
}

extern "C" int pg_delta_prep(float* rec, const void* proj, int ld, int r_col0, int k_col0, int v_col0, int a_col0,
                             int lora_col0, int lora, const void* w2, const void* w0, const void* a_bias, int n_tokens,
                             int heads, int dim, float decay_scale, float key_eps, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(rec && proj && w2 && w0 && lora > 0 && heads > 0 && dim > 0, "delta_prep: bad arguments");
  const size_t smem = sizeof(float) * PREP_TOK * ((size_t)lora + heads);
  PG_DISPATCH_DTYPE(dtype, T, {
    const int threads = heads * dim >= 256 ? 256 : 128;
    const int slices = n_tokens <= 64 ? cdiv(heads * dim, threads) : 1;
    return launch_pdl("delta_prep", delta_prep_kernel<T>, dim3(cdiv(n_tokens, PREP_TOK), slices), dim3(threads),
                      smem, (cudaStream_t)stream, rec, (const T*)proj, ld, r_col0, k_col0, v_col0, a_col0, lora_col0, lora,
                      (const T*)w2, (const T*)w0, (const T*)a_bias, n_tokens, heads, dim, (dim + 3) / 4 * 4, decay_scale,
                      key_eps);
  });
  return PG_OK;
}

extern "C" int pg_delta_rule(float* out, float* state, const float* rec, const int32_t* segs, int n_segs, int heads,
                             int dim, void* stream) {
  if (n_segs <= 0) return PG_OK;
  PG_REQUIRE(out && state && rec && segs, "delta_rule: bad arguments");
  PG_REQUIRE(dim > 0 && dim <= 256, "delta_rule: head size %d (1..256)", dim);
  cudaStream_t st = (cudaStream_t)stream;
  if (dim <= 32) return launch_delta<32, 8>(out, state, rec, segs, n_segs, heads, dim, st);
  if (dim <= 64) return launch_delta<64, 8>(out, state, rec, segs, n_segs, heads, dim, st);
  if (dim <= 128) return launch_delta<128, 4>(out, state, rec, segs, n_segs, heads, dim, st);
  return launch_delta<256, 2>(out, state, rec, segs, n_segs, heads, dim, st);
}

extern "C" int pg_headnorm_gate(void* out, int ld_out, const float* o, const void* w, const void* gate, int ld_gate,
                                int n_tokens, int heads, int dim, float eps, float out_scale, int dtype, void* stream) {
  return pg_headnorm_gate_ex(out, ld_out, o, w, gate, ld_gate, 0, n_tokens, heads, dim, eps, out_scale, dtype, stream);
}

extern "C" int pg_headnorm_gate_ex(void* out, int ld_out, const float* o, const void* w, const void* gate, int ld_gate,
                                   int gate_silu, int n_tokens, int heads, int dim, float eps, float out_scale, int dtype,
                                   void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(out && o && heads > 0 && dim > 0, "headnorm_gate: bad arguments");
  const int warps = 8;
  const int pairs = (dim % 2 == 0 && ld_out % 2 == 0 && ld_gate % 2 == 0 && ((uintptr_t)out % 4) == 0 &&
                     ((uintptr_t)o % 8) == 0) ? 1 : 0;
  PG_DISPATCH_DTYPE(dtype, T, {
    return launch_pdl("headnorm_gate", headnorm_gate_kernel<T>, dim3(cdiv((long long)n_tokens * heads, warps)),
                      dim3(warps * 32), 0, (cudaStream_t)stream, (T*)out, ld_out, o, (const T*)w, (const T*)gate, ld_gate,
                      n_tokens, heads, dim, eps, out_scale, pairs, gate_silu ? 1 : 0);
  });
  return PG_OK;
}

extern "C" long long pg_lightning_record_floats(int n_tokens, int heads, int dim, int vdim) {
  return (long long)n_tokens * heads * (2 * ((dim + 3) / 4 * 4) + (vdim + 3) / 4 * 4);
}

extern "C" int pg_lightning_prep(float* rec, const void* proj, int ld, int q_col0, int k_col0, int v_col0, int n_tokens,
                                 int heads, int dim, int vdim, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(rec && proj && heads > 0 && dim > 0 && vdim > 0, "lightning_prep: bad arguments");
  const int dp = (dim + 3) / 4 * 4, vp = (vdim + 3) / 4 * 4;
  PG_DISPATCH_DTYPE(dtype, T, {
    constexpr int V = Vec<T>::N;
    if (dim % V == 0 && vdim % V == 0 && ld % V == 0 && q_col0 % V == 0 && k_col0 % V == 0 && v_col0 % V == 0 &&
        (((uintptr_t)proj | (uintptr_t)rec) & 15) == 0) {
      const int vecs = heads * (2 * dim + vdim) / V, threads = vecs >= 256 ? 256 : (vecs + 31) / 32 * 32;
      return launch_pdl("lightning_prep", lightning_prep_vec_kernel<T>, dim3(n_tokens), dim3(threads), 0, (cudaStream_t)stream, rec,
                        (const T*)proj, ld, q_col0, k_col0, v_col0, heads, dim, vdim);
    }
    return launch_pdl("lightning_prep", lightning_prep_kernel<T>, dim3(n_tokens), dim3(256), 0, (cudaStream_t)stream, rec,
                      (const T*)proj, ld, q_col0, k_col0, v_col0, (long long)n_tokens, heads, dim, vdim, dp, vp);
  });
  return PG_OK;
}

extern "C" int pg_retention_prep(float* rec, const void* proj, int ld, int q_col0, int k_col0, int v_col0, const float* freq,
                                 int rot_dims, int interleaved, float k_scale, const int32_t* tok_pos, int n_tokens, int heads,
                                 int dim, int vdim, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(rec && proj && tok_pos && heads > 0 && dim > 0 && vdim > 0, "retention_prep: bad arguments");
  PG_REQUIRE(rot_dims >= 0 && rot_dims <= dim && rot_dims % 2 == 0 && (rot_dims == 0 || freq),
             "retention_prep: %d rotated columns of %d (even, with a frequency table)", rot_dims, dim);
  const int dp = (dim + 3) / 4 * 4, vp = (vdim + 3) / 4 * 4;
  const int work = heads * (2 * dp + vp) / 4, threads = work >= 512 ? 256 : (work >= 128 ? 128 : 64);
  PG_DISPATCH_DTYPE(dtype, T, {
    return launch_pdl("retention_prep", retention_prep_kernel<T>, dim3(n_tokens), dim3(threads), sizeof(float) * (size_t)rot_dims,
                      (cudaStream_t)stream, rec, (const T*)proj, ld, q_col0, k_col0, v_col0, (const float2*)freq, rot_dims,
                      interleaved ? 1 : 0, k_scale, tok_pos, heads, dim, vdim, dp, vp);
  });
  return PG_OK;
}

extern "C" int pg_lightning_attention(float* out, float* state, const float* rec, const float* decay, const int32_t* segs,
                                      int n_segs, int heads, int dim, int vdim, void* stream) {
  return pg_lightning_attention_ex(out, state, rec, decay, nullptr, segs, n_segs, heads, dim, vdim, stream);
}

static int lightning_any(float* out, float* state, const float* rec, const float* decay, const float* skip, int td,
                         const int32_t* segs, int n_segs, int heads, int dim, int vdim, int no_wait, int* err, void* stream) {
  if (n_segs <= 0) return PG_OK;
  PG_REQUIRE(out && state && rec && segs, "lightning_attention: bad arguments");
  PG_REQUIRE(dim > 0 && dim <= 256 && vdim > 0, "lightning_attention: key size %d (1..256), value size %d", dim, vdim);
  cudaStream_t st = (cudaStream_t)stream;
  // lanes per value column: a thread keeps DMAX / RG rows of the state
  if (dim <= 32) return launch_scan<32>(out, state, rec, decay, skip, td, segs, n_segs, heads, dim, vdim, no_wait, err, st);
  if (dim <= 64) return launch_scan<64>(out, state, rec, decay, skip, td, segs, n_segs, heads, dim, vdim, no_wait, err, st);
  if (dim <= 128) return launch_scan<128>(out, state, rec, decay, skip, td, segs, n_segs, heads, dim, vdim, no_wait, err, st);
  return launch_scan<256>(out, state, rec, decay, skip, td, segs, n_segs, heads, dim, vdim, no_wait, err, st);
}

extern "C" int pg_lightning_attention_ex(float* out, float* state, const float* rec, const float* decay, const float* skip,
                                         const int32_t* segs, int n_segs, int heads, int dim, int vdim, void* stream) {
  // no constant decay: the records carry one per token
  return lightning_any(out, state, rec, decay, skip, decay ? DECAY_HEAD : DECAY_TOKEN, segs, n_segs, heads, dim, vdim, 0, nullptr, stream);
}

extern "C" int pg_gla_attention(float* out, float* state, const float* rec, const int32_t* segs, int n_segs, int heads, int dim,
                                int vdim, void* stream) {
  return lightning_any(out, state, rec, nullptr, nullptr, DECAY_CHANNEL, segs, n_segs, heads, dim, vdim, 0, nullptr, stream);
}

extern "C" int pg_linear_scan(float* out, float* state, const float* rec, const float* decay, const float* skip, int per_channel,
                              const int32_t* segs, int n_segs, int heads, int dim, int vdim, int no_wait, int* err_flag, void* stream) {
  PG_REQUIRE(!per_channel || (!decay && !skip), "linear_scan: a decay per channel lies in the records and goes without a direct term");
  return lightning_any(out, state, rec, decay, skip, per_channel ? DECAY_CHANNEL : (decay ? DECAY_HEAD : DECAY_TOKEN), segs, n_segs,
                       heads, dim, vdim, no_wait, err_flag, stream);
}

extern "C" long long pg_gla_record_floats(int n_tokens, int heads, int dim, int vdim) {
  return (long long)n_tokens * heads * (3 * ((dim + 3) / 4 * 4) + (vdim + 3) / 4 * 4);
}

extern "C" int pg_gla_prep(float* rec, const void* proj, int ld, int q_col0, int k_col0, int v_col0, int a_col0, int rank,
                           const void* w2, const void* b2, float q_scale, float inv_tau, int n_tokens, int heads, int dim,
                           int vdim, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_REQUIRE(rec && proj && w2 && b2 && rank > 0 && heads > 0 && dim > 0 && vdim > 0, "gla_prep: bad arguments");
  const int dp = (dim + 3) / 4 * 4, vp = (vdim + 3) / 4 * 4;
  const size_t smem = sizeof(float) * PREP_TOK * (size_t)rank;
  PG_REQUIRE(smem <= 200 * 1024, "gla_prep: an inner projection of %d columns does not fit shared memory", rank);
  PG_DISPATCH_DTYPE(dtype, T, {
    const int work = heads * (dp > vp ? dp : vp), threads = work >= 256 ? 256 : 128;
    const int slices = n_tokens <= 64 ? cdiv(heads * dp, threads) : 1;
    return launch_pdl("gla_prep", gla_prep_kernel<T>, dim3(cdiv(n_tokens, PREP_TOK), slices), dim3(threads), smem,
                      (cudaStream_t)stream, rec, (const T*)proj, ld, q_col0, k_col0, v_col0, a_col0, rank, (const T*)w2,
                      (const T*)b2, q_scale, inv_tau, n_tokens, heads, dim, vdim, dp, vp);
  });
  return PG_OK;
}
