// Decode attention: one new token per sequence against the paged KV cache
// (reference GemmaAttention.forward q_len==1, modeling_gemma.py:262-288; mask all zeros, fp32
// softmax).  The G query heads of a KV head share every K/V load (repeat_kv, :136-141, is never
// materialised).
//
// One thread-block cluster of DC_NS CTAs per (sequence, kv head): the cluster's DC_NS*8 warps
// take the cached tokens round-robin, each warp loads K and V rows for a batch of tokens at once
// (all loads in flight before the first use), keeps a flash-style (m, l, acc) per head in
// registers, the warps of a CTA merge through shared memory and the CTAs of the cluster merge
// through distributed shared memory — no global workspace, no atomics, one launch.
// Work is tiny (T*1 KB per layer); the design goal is latency, not bandwidth.
//
// 16-bit models with head_dim 256 and up to 8 query heads per KV head take decode_attention_mma_kernel instead (below).
#include <cmath>
#include <cooperative_groups.h>

#include "common.cuh"
#include "mma_frag.cuh"

namespace cg = cooperative_groups;

namespace pg {

constexpr int DC_WARPS = 8;     // warps per CTA
constexpr int DC_MAX_PT = 1024; // page-table entries staged in shared memory

template <typename T, int G, int NCH, int TB, int DC_NS>
__global__ void __launch_bounds__(DC_WARPS * 32, 1)
decode_attention_cluster_kernel(T* __restrict__ out, const T* __restrict__ q, const T* __restrict__ k_pool,
                                const T* __restrict__ v_pool, const int32_t* __restrict__ page_table,
                                int pt_stride, int page_size, const int32_t* __restrict__ kv_len,
                                int kv_len_add, int nq, int nkv, int hd, float scale_div, float scale_mul,
                                Prefetch pf) {
  constexpr int V = Vec<T>::N;
  cg::cluster_group cluster = cg::this_cluster();
  pdl_launch_dependents();
  l2_prefetch_slice(pf);
  const int rank = (int)cluster.block_rank();
  const int b = blockIdx.y, kvh = blockIdx.z;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  pdl_wait();  // q and this step's K/V row come from the preceding qkv kernel
  const int T_len = kv_len[b] + kv_len_add;
  const int row_elems = nkv * hd;

  extern __shared__ __align__(16) float sm[];
  float* s_acc = sm;                                     // [DC_WARPS][G][hd]
  float* s_m = s_acc + (size_t)DC_WARPS * G * hd;        // [DC_WARPS][G]
  float* s_l = s_m + DC_WARPS * G;                       // [DC_WARPS][G]
  float* c_acc = s_l + DC_WARPS * G;                     // [G][hd]   CTA-level partial (read by peers)
  float* c_m = c_acc + (size_t)G * hd;                   // [G]
  float* c_l = c_m + G;                                  // [G]
  __shared__ int s_pt[DC_MAX_PT];

  const int n_pages = (T_len + page_size - 1) / page_size;
  const bool pt_in_smem = n_pages <= DC_MAX_PT;
  if (pt_in_smem)
    for (int i = threadIdx.x; i < n_pages; i += DC_WARPS * 32) s_pt[i] = page_table[(size_t)b * pt_stride + i];

  float qf[G][NCH][V];
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int d = (c * 32 + lane) * V;
      if (d < hd) unpack<T>(ldg_cached(q + (size_t)b * nq * hd + (size_t)(kvh * G + g) * hd + d), qf[g][c]);
      else
#pragma unroll
        for (int i = 0; i < V; ++i) qf[g][c][i] = 0.f;
    }
  float m[G], l[G], acc[G][NCH][V];
  float m_run = -INFINITY, l_run = 0.f;   // transposed path: lane L keeps the state of head L % G
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY; l[g] = 0.f;
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[g][c][i] = 0.f;
  }
  __syncthreads();

  constexpr int NW = DC_NS * DC_WARPS;
  const int gw = rank * DC_WARPS + wid;
  for (int j0 = gw; j0 < T_len; j0 += NW * TB) {
    uint4 kr[TB][NCH], vr[TB][NCH];
#pragma unroll
    for (int t = 0; t < TB; ++t) {
      const int j = j0 + t * NW;
      if (j < T_len) {
        const int page = pt_in_smem ? s_pt[j / page_size] : page_table[(size_t)b * pt_stride + j / page_size];
        const size_t row = ((size_t)page * page_size + (j % page_size)) * (size_t)row_elems + (size_t)kvh * hd;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          const int d = (c * 32 + lane) * V;
          if (d < hd) { kr[t][c] = ldg_cached(k_pool + row + d); vr[t][c] = ldg_cached(v_pool + row + d); }
          else { kr[t][c] = make_uint4(0, 0, 0, 0); vr[t][c] = make_uint4(0, 0, 0, 0); }
        }
      } else {
#pragma unroll
        for (int c = 0; c < NCH; ++c) { kr[t][c] = make_uint4(0, 0, 0, 0); vr[t][c] = make_uint4(0, 0, 0, 0); }
      }
    }
    float s[TB][G];
#pragma unroll
    for (int t = 0; t < TB; ++t) {
      float kf[NCH][V];
#pragma unroll
      for (int c = 0; c < NCH; ++c) unpack<T>(kr[t][c], kf[c]);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float a = 0.f;
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
          for (int i = 0; i < V; ++i) a = fmaf(qf[g][c][i], kf[c][i], a);
        s[t][g] = a;
      }
    }
    if constexpr (TB * G == 32) {
      // 32 (token, head) partial dots per lane -> transposed butterfly: 31 shuffles leave lane L with the full
      // sum of pair L = t*G + g (instead of 32 x 5 shuffles with every lane holding every sum), so the scale /
      // max / exp work is done once per pair, not 32 times.
      float sv[32];
#pragma unroll
      for (int t = 0; t < TB; ++t)
#pragma unroll
        for (int g = 0; g < G; ++g) sv[t * G + g] = s[t][g];
#pragma unroll
      for (int w = 16; w >= 1; w >>= 1) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; ++i) {
          const float keep = up ? sv[i + w] : sv[i];
          const float send = up ? sv[i] : sv[i + w];
          sv[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
      }
      const int my_t = lane / G;
      // matmul output rounded to the model dtype, then "/ sqrt(head_dim)" (modeling_gemma.py:266); a power-of-two
      // divisor is applied as an exact multiply (same bits, no division routine)
      const float sr = rnd<T>(sv[0]);
      float sc = (scale_mul != 0.f) ? sr * scale_mul : rnd<T>(sr / scale_div);
      sc = (j0 + my_t * NW < T_len) ? sc : -INFINITY;
      float mx = sc;
#pragma unroll
      for (int o = G; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));  // over the TB tokens of my head
      const float mn = fmaxf(m_run, mx);
      const float corr = __expf(m_run - mn);
      const float pr = __expf(sc - mn);                      // 0 for padded tokens
      float psum = pr;
#pragma unroll
      for (int o = G; o < 32; o <<= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
      m_run = mn;
      l_run = l_run * corr + psum;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float cg = __shfl_sync(0xffffffffu, corr, g);
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
          for (int i = 0; i < V; ++i) acc[g][c][i] *= cg;
      }
#pragma unroll
      for (int t = 0; t < TB; ++t) {
        float vf[NCH][V];
#pragma unroll
        for (int c = 0; c < NCH; ++c) unpack<T>(vr[t][c], vf[c]);
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float pg = __shfl_sync(0xffffffffu, pr, t * G + g);
#pragma unroll
          for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int i = 0; i < V; ++i) acc[g][c][i] = fmaf(pg, vf[c][i], acc[g][c][i]);
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < TB; ++t)
  #pragma unroll
        for (int g = 0; g < G; ++g) s[t][g] = warp_sum(s[t][g]);
  #pragma unroll
      for (int g = 0; g < G; ++g) {
        float mn = m[g];
  #pragma unroll
        for (int t = 0; t < TB; ++t) {
          // matmul output rounded to the model dtype, then "/ sqrt(head_dim)" (modeling_gemma.py:266)
          // (a power-of-two divisor is applied as an exact multiply: same bits, no division routine)
          const float sr = rnd<T>(s[t][g]);
          const float sc = (scale_mul != 0.f) ? sr * scale_mul : rnd<T>(sr / scale_div);
          s[t][g] = (j0 + t * NW < T_len) ? sc : -INFINITY;
          mn = fmaxf(mn, s[t][g]);
        }
        const float corr = __expf(m[g] - mn);
        m[g] = mn;
        l[g] *= corr;
  #pragma unroll
        for (int c = 0; c < NCH; ++c)
  #pragma unroll
          for (int i = 0; i < V; ++i) acc[g][c][i] *= corr;
  #pragma unroll
        for (int t = 0; t < TB; ++t) s[t][g] = __expf(s[t][g] - mn);  // p; 0 for the padded tokens
  #pragma unroll
        for (int t = 0; t < TB; ++t) l[g] += s[t][g];
      }
  #pragma unroll
      for (int t = 0; t < TB; ++t) {
        float vf[NCH][V];
  #pragma unroll
        for (int c = 0; c < NCH; ++c) unpack<T>(vr[t][c], vf[c]);
  #pragma unroll
        for (int g = 0; g < G; ++g)
  #pragma unroll
          for (int c = 0; c < NCH; ++c)
  #pragma unroll
            for (int i = 0; i < V; ++i) acc[g][c][i] = fmaf(s[t][g], vf[c][i], acc[g][c][i]);
      }
    }
  }
  if constexpr (TB * G == 32) {  // the per-head running (m, l) live in the lanes of that head: gather them
#pragma unroll
    for (int g = 0; g < G; ++g) { m[g] = __shfl_sync(0xffffffffu, m_run, g); l[g] = __shfl_sync(0xffffffffu, l_run, g); }
  }

  // ---- merge the warps of this CTA
#pragma unroll
  for (int g = 0; g < G; ++g) {
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int d = (c * 32 + lane) * V;
      if (d < hd)
#pragma unroll
        for (int i = 0; i < V; i += 4)
          *reinterpret_cast<float4*>(&s_acc[((size_t)wid * G + g) * hd + d + i]) =
              make_float4(acc[g][c][i], acc[g][c][i + 1], acc[g][c][i + 2], acc[g][c][i + 3]);
    }
    if (lane == 0) { s_m[wid * G + g] = m[g]; s_l[wid * G + g] = l[g]; }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < G * hd; e += DC_WARPS * 32) {
    const int g = e / hd, d = e % hd;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) M = fmaxf(M, s_m[w * G + g]);
    float a = 0.f;
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) {
      const float mw = s_m[w * G + g];
      if (mw != -INFINITY) a = fmaf(__expf(mw - M), s_acc[((size_t)w * G + g) * hd + d], a);
    }
    c_acc[e] = a;
  }
  if (threadIdx.x < G) {
    const int g = threadIdx.x;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) M = fmaxf(M, s_m[w * G + g]);
    float L = 0.f;
#pragma unroll
    for (int w = 0; w < DC_WARPS; ++w) {
      const float mw = s_m[w * G + g];
      if (mw != -INFINITY) L = fmaf(__expf(mw - M), s_l[w * G + g], L);
    }
    c_m[g] = M;
    c_l[g] = L;
  }
  cluster.sync();  // every CTA's partial is visible cluster-wide

  // ---- merge the CTAs: CTA `rank` finalises its slice of the G*hd outputs through DSMEM
  const int per = (G * hd + DC_NS - 1) / DC_NS;
  const int e_end = min(G * hd, (rank + 1) * per);
  for (int e = rank * per + threadIdx.x; e < e_end; e += DC_WARPS * 32) {
    const int g = e / hd;
    float pm[DC_NS], pl[DC_NS], pa[DC_NS];
#pragma unroll
    for (int r = 0; r < DC_NS; ++r) {
      pm[r] = *cluster.map_shared_rank(c_m + g, r);
      pl[r] = *cluster.map_shared_rank(c_l + g, r);
      pa[r] = *cluster.map_shared_rank(c_acc + e, r);
    }
    float M = -INFINITY;
#pragma unroll
    for (int r = 0; r < DC_NS; ++r) M = fmaxf(M, pm[r]);
    float a = 0.f, L = 0.f;
#pragma unroll
    for (int r = 0; r < DC_NS; ++r)
      if (pm[r] != -INFINITY) {
        const float w = __expf(pm[r] - M);
        a = fmaf(w, pa[r], a);
        L = fmaf(w, pl[r], L);
      }
    out[(size_t)b * nq * hd + (size_t)(kvh * G + g) * hd + (e % hd)] = from_f<T>(a / L);
  }
  cluster.sync();  // nobody leaves while a peer may still read its shared memory
}

// x / 2^k == x * 2^-k exactly (no underflow at these magnitudes): skip the IEEE division routine
static float exact_reciprocal(float scale_div) {
  int ex = 0;
  return (frexpf(scale_div, &ex) == 0.5f) ? 1.0f / scale_div : 0.f;
}

template <typename T, int G, int NCH, int DC_NS>
static int launch_da_ns(void* out, const void* q, const void* k_pool, const void* v_pool, const int32_t* page_table,
                     int pt_stride, int page_size, const int32_t* kv_len, int kv_len_add, int B, int nq, int nkv,
                     int hd, float scale_div, Prefetch pf, cudaStream_t st) {
  constexpr int TB = NCH == 1 ? 4 : 2;
  auto kern = decode_attention_cluster_kernel<T, G, NCH, TB, DC_NS>;
  if (DC_NS > 8) cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  const float scale_mul = exact_reciprocal(scale_div);
  const size_t smem = ((size_t)DC_WARPS * G * hd + 2 * DC_WARPS * G + (size_t)G * hd + 2 * G) * sizeof(float);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    set_error("decode_attention: cannot reserve %zu B of shared memory", smem);
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(DC_NS, B, nkv);
  cfg.blockDim = dim3(DC_WARPS * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  static const int pdl = env_int("PG_PDL", 1);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = DC_NS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (T*)out, (const T*)q, (const T*)k_pool, (const T*)v_pool,
                                     page_table, pt_stride, page_size, kv_len, kv_len_add, nq, nkv, hd, scale_div,
                                     scale_mul, pf);
  if (e != cudaSuccess) {
    set_error("decode_attention launch: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  return check_launch("decode_attention");
}

template <typename T, int G, int NCH>
static int launch_da(void* out, const void* q, const void* k_pool, const void* v_pool, const int32_t* page_table,
                     int pt_stride, int page_size, const int32_t* kv_len, int kv_len_add, int B, int nq, int nkv,
                     int hd, float scale_div, Prefetch pf, cudaStream_t st) {
  // Cluster size: as many CTAs per (sequence, kv head) as keeps the whole launch within one wave of the 148 SMs
  // (the kernel needs a full SM: 255 registers x 256 threads).  16 is a non-portable cluster size.
  static const int ns_env = env_int("PG_ATTN_NS", 0);
  int ns = ns_env;
  if (!ns) {
    const int seqs = B * nkv;
    ns = seqs <= 9 ? 16 : (seqs <= 18 ? 8 : (seqs <= 37 ? 4 : (seqs <= 74 ? 2 : 1)));
  }
#define PG_DA_NS(N_) \
  return launch_da_ns<T, G, NCH, N_>(out, q, k_pool, v_pool, page_table, pt_stride, page_size, kv_len, kv_len_add, B, nq, nkv, hd, scale_div, pf, st)
  switch (ns) {
    case 16: PG_DA_NS(16);
    case 8: PG_DA_NS(8);
    case 4: PG_DA_NS(4);
    case 2: PG_DA_NS(2);
    default: PG_DA_NS(1);
  }
#undef PG_DA_NS
}

// ------------------------------------------------------------------------------------------------ head_dim 256 on mma.sync
// The kernel above is bound by its chain, not by bytes: 255 registers x 256 threads fill an SM, so a cluster of 16 CTAs needs 16
// free SMs of one GPC (8 sequences do not fit at once: 1345 cached tokens took 39.7 us for 11 MB), and every token costs a
// warp 8 x 16 FMAs plus a 31-shuffle butterfly.  Here the 8 query heads are the N dimension of mma.m16n8k16:
//   S^T [16 tokens x 8 heads] = K Q^T     A = 16 key rows,   B = the query rows
//   O^T [256 dims x 8 heads] += V^T P^T   A = V transposed,  B = the weights
// A warp takes 16 tokens at a time and all operands go from global memory straight into fragments with 16-byte loads: the
// contraction index of S^T is permuted (lane j of a quad owns 8 consecutive columns of every 32) and so are the rows of O^T
// (lane group r owns 8 consecutive columns of every 64), which neither product notices.  The weights stay fp32: they enter
// as three 16-bit terms (mma_frag.cuh; all their 24 bits in bf16, 2^-39 of the largest weight in fp16); only QK^T's operands are
// 16-bit, as stored.  128 threads per CTA and two CTAs per SM keep a cluster of 16 within 8 SMs.
// Measured (launch alone, cold cache): 1 sequence x 262 tokens 13.5 -> 9.5 us, 8 x 1345 39.7 -> 14.2 us, 32 x 389 23.6 -> 12.1 us;
// inside the captured step 4.0, 23 and 5.1 us per layer less.
// What then bounded it was the tail, 4 to 5 us of 7 to 11 behind the wait: merging the warps (1.6 to 2.8 us), fetching the peers' sums
// (1.7) and the barrier behind that (0.75).  With the sums handed over by the CTAs that have them, and the rows in L2 before the wait,
// behind the wait: 1 sequence x 262 tokens 7.0 -> 4.9 us, 8 x 1345 11.3 -> 7.9, 32 x 389 10.5 -> 6.7.
// (The next chunk's keys requested behind this one's scores: 48 bytes spilled, and no faster.)
constexpr int DM_WARPS = 4, DM_HD = 256, DM_G = 8;

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" :: "l"(p)); }

// ROPE: the step's rotary embedding and cache row too.  q is then the q/k/v projections [B][nq + 2 nkv][256]: every CTA rotates its
// heads' query rows (pg_rope_append's arithmetic and rounding) into shared memory, and the one that meets the last chunk writes the
// new key and value row before it reads the chunk.  As a launch of its own that was 4.3 us for 8 rows of 10 heads, most of it the
// launch and the chain position -> page -> load -> store; here the loads go out with those of the length and the pages and the angles
// are there before the wait.  Six layers: 8 sequences x 1345 tokens 406 -> 402 us, 32 x 389 452 -> 437; the two launches stay for
// what this kernel does not take.
struct DecodeRope {
  const float* inv_freq;
  const int32_t* positions;
  int max_pos;
};

template <typename T, int NS, bool ROPE, bool AHEAD>
__global__ void __launch_bounds__(DM_WARPS * 32, 2)
decode_attention_mma_kernel(T* __restrict__ out, const T* __restrict__ q, const T* k_pool, const T* v_pool,
                            const int32_t* __restrict__ page_table, int pt_stride, int page_size, int num_pages,
                            const int32_t* __restrict__ kv_len, int kv_len_add, int nq, int nkv, float scale_div,
                            float scale_mul, DecodeRope rope, Prefetch pf) {
  constexpr int KB = DM_HD / 32, VB = DM_HD / 64;
  cg::cluster_group cluster = cg::this_cluster();
  pdl_launch_dependents();
  l2_prefetch_slice(pf);
  const int rank = (int)cluster.block_rank(), b = blockIdx.y, kvh = blockIdx.z, G = nq / nkv;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, r = lane >> 2, j = lane & 3;
  __shared__ __align__(16) float s_acc[DM_WARPS][DM_G][DM_HD + 4];
  // what the cluster's CTAs have put here for this CTA's share of the outputs: [CTA][output of the share], [CTA][head]{maximum, sum}
  __shared__ __align__(16) float r_acc[DM_G * DM_HD];
  __shared__ float2 r_ml[NS][DM_G];
  __shared__ float s_m[DM_WARPS][DM_G], s_l[DM_WARPS][DM_G];
  __shared__ int s_pt[DC_MAX_PT];
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // waited for before anything goes to another CTA
  const int32_t* pt = page_table + (size_t)b * pt_stride;
  const size_t row_elems = (size_t)nkv * DM_HD;
  // While the preceding kernel runs (1.5 to 2.5 us in a captured step): this warp's first four chunks into L2.  A hint only: the length
  // and the page numbers it goes by are read again behind the wait.  The preceding kernel may be about to write them, so a number
  // names an address only if the pool has that page; where the caller did not say how many it has (!AHEAD), nothing is asked for.
  const int jp = threadIdx.x & 63;
  int ahead[4], t_end = 0;
  if constexpr (AHEAD) {
#pragma unroll
    for (int i = 0; i < 4; ++i) ahead[i] = __ldcg(pt + min((rank + NS * (wid + DM_WARPS * i)) * 16 / page_size, pt_stride - 1));
    t_end = __ldcg(kv_len + b) + kv_len_add;
  }
  // ... and the angles of this thread's columns 2 jp, 2 jp + 1, done again if what they come from is another behind the wait
  float angle[2] = {0.f, 0.f}, c[2], s[2];
  auto angles = [&] {
    const float pos = (float)min(max(__ldcg(rope.positions + b), 0), rope.max_pos - 1);
    const float2 f = __ldcg(reinterpret_cast<const float2*>(rope.inv_freq) + jp);
    const float a0 = pos * f.x, a1 = pos * f.y;
    const bool other = a0 != angle[0] || a1 != angle[1];
    angle[0] = a0; angle[1] = a1;
    return other;
  };
  if constexpr (ROPE) angles();
  if constexpr (AHEAD) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = (rank + NS * (wid + DM_WARPS * i)) * 16 + (lane >> 1);
      if (t >= t_end || (unsigned)ahead[i] >= (unsigned)num_pages) break;
      const size_t at = ((size_t)ahead[i] * page_size + t % page_size) * row_elems + (size_t)kvh * DM_HD + (lane & 1) * 128;
      prefetch_l2(k_pool + at);
      prefetch_l2(k_pool + at + 64);
      prefetch_l2(v_pool + at);
      prefetch_l2(v_pool + at + 64);
    }
  }
  if constexpr (ROPE) {
#pragma unroll
    for (int i = 0; i < 2; ++i) { c[i] = rnd<T>(cosf(angle[i])); s[i] = rnd<T>(sinf(angle[i])); }
  }
  pdl_wait();  // q and this step's K/V row come from the preceding qkv kernel

  // the length, the page-table row and the query rows are requested together
  const int T_len = kv_len[b] + kv_len_add;
  const int pt_n = min(pt_stride, DC_MAX_PT);
  for (int i = threadIdx.x; i < pt_n; i += DM_WARPS * 32) s_pt[i] = pt[i];
  uint4 qf[KB];
  if constexpr (ROPE) {
    typedef uint32_t u32;
    constexpr int LD = DM_HD + 32, HALF = DM_HD / 2;          // rows of 144 words: the fragments' 16-byte reads meet no bank twice
    T* s_q = reinterpret_cast<T*>(s_acc);                     // until the sums need the room
    const int slot = T_len - 1;
    const T* row = q + (size_t)b * (nq + 2 * nkv) * DM_HD;
    const bool newest = (slot / 16) % NS == rank;             // this CTA meets the last chunk
    u32 lo[DM_G / 2 + 1], hi[DM_G / 2 + 1];
#pragma unroll
    for (int i = 0; i <= DM_G / 2; ++i) {                      // its query heads, then the key head
      const int h = min(2 * i + (int)(threadIdx.x >> 6), G);
      const T* at = row + (size_t)(h < G ? kvh * G + h : nq + kvh) * DM_HD + 2 * jp;
      lo[i] = __ldg(reinterpret_cast<const u32*>(at));
      hi[i] = __ldg(reinterpret_cast<const u32*>(at + HALF));
    }
    const u32 nv = __ldg(reinterpret_cast<const u32*>(row + (size_t)(nq + nkv + kvh) * DM_HD + 2 * threadIdx.x));
    if (angles()) {
#pragma unroll
      for (int i = 0; i < 2; ++i) { c[i] = rnd<T>(cosf(angle[i])); s[i] = rnd<T>(sinf(angle[i])); }
    }
    u32 nk_lo = 0, nk_hi = 0;
#pragma unroll
    for (int i = 0; i <= DM_G / 2; ++i) {
      const int h = 2 * i + (threadIdx.x >> 6);
      if (h > G) continue;
      float x[2], y[2];
      unpack_pair<T>(lo[i], x);
      unpack_pair<T>(hi[i], y);
      const u32 l2 = pack_pair<T>(rnd<T>(x[0] * c[0]) + rnd<T>(-y[0] * s[0]), rnd<T>(x[1] * c[1]) + rnd<T>(-y[1] * s[1]));
      const u32 h2 = pack_pair<T>(rnd<T>(y[0] * c[0]) + rnd<T>(x[0] * s[0]), rnd<T>(y[1] * c[1]) + rnd<T>(x[1] * s[1]));
      if (h == G) { nk_lo = l2; nk_hi = h2; continue; }
      *reinterpret_cast<u32*>(s_q + h * LD + 2 * jp) = l2;
      *reinterpret_cast<u32*>(s_q + h * LD + HALF + 2 * jp) = h2;
    }
    __syncthreads();
    if (newest) {
      const int pi = slot / page_size, page = pi < pt_n ? s_pt[pi] : pt[pi];
      const size_t at = ((size_t)page * page_size + slot % page_size) * row_elems + (size_t)kvh * DM_HD;
      if ((threadIdx.x >> 6) == (G & 1)) {
        *reinterpret_cast<u32*>(const_cast<T*>(k_pool) + at + 2 * jp) = nk_lo;
        *reinterpret_cast<u32*>(const_cast<T*>(k_pool) + at + HALF + 2 * jp) = nk_hi;
      }
      *reinterpret_cast<u32*>(const_cast<T*>(v_pool) + at + 2 * threadIdx.x) = nv;
    }
#pragma unroll
    for (int kb = 0; kb < KB; ++kb)
      qf[kb] = r < G ? *reinterpret_cast<const uint4*>(s_q + r * LD + kb * 32 + j * 8) : make_uint4(0, 0, 0, 0);
  } else {
    const T* qr = q + ((size_t)b * nq + (size_t)kvh * G + r) * DM_HD + j * 8;
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) qf[kb] = r < G ? ldg_cached(qr + kb * 32) : make_uint4(0, 0, 0, 0);
  }
  float acc[VB][4][4], m[2], l[2];                          // m, l: heads 2j and 2j + 1, the same in every lane group
  __syncthreads();

  const int chunks = (T_len + 15) / 16;
  auto load_row = [](const T* p) {                            // ROPE: the last row is this kernel's own
    if constexpr (ROPE) return __ldcg(reinterpret_cast<const uint4*>(p));
    else return ldg_cached(p);
  };
  auto attend = [&](auto in_fp32) {                           // this warp's chunks
    constexpr bool fp32 = decltype(in_fp32)::value;
#pragma unroll
    for (int vb = 0; vb < VB; ++vb)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[vb][i][e] = 0.f;
    m[0] = m[1] = -INFINITY;
    l[0] = l[1] = 0.f;
    // chunk c: CTA c % NS first, so that a short context spreads over the SMs before it stacks up in one
    for (int c = rank + NS * wid; c < chunks; c += NS * DM_WARPS) {
      const int t0 = c * 16, pi = t0 / page_size;               // page_size is a multiple of 16: one page per chunk
      const int page = pi < pt_n ? s_pt[pi] : pt[pi];
      const size_t base = ((size_t)page * page_size + t0 % page_size) * row_elems + (size_t)kvh * DM_HD;
      const int last = T_len - 1 - t0;                          // rows behind the last token repeat it with weight 0
      const T* kp = k_pool + base + j * 8;
      const T* vp = v_pool + base + r * 8;
      const size_t k0 = (size_t)min(r, last) * row_elems, k1 = (size_t)min(r + 8, last) * row_elems;
      const size_t v0 = (size_t)min(2 * j, last) * row_elems, v1 = (size_t)min(2 * j + 1, last) * row_elems;
      const size_t v2 = (size_t)min(2 * j + 8, last) * row_elems, v3 = (size_t)min(2 * j + 9, last) * row_elems;
      uint4 ka[KB], kc[KB], va[VB][4];
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) { ka[kb] = load_row(kp + k0 + kb * 32); kc[kb] = load_row(kp + k1 + kb * 32); }
#pragma unroll
      for (int vb = 0; vb < VB; ++vb) {
        va[vb][0] = load_row(vp + v0 + vb * 64); va[vb][1] = load_row(vp + v1 + vb * 64);
        va[vb][2] = load_row(vp + v2 + vb * 64); va[vb][3] = load_row(vp + v3 + vb * 64);
      }
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) {
        mma_16816<T>(s0, ka[kb].x, kc[kb].x, ka[kb].y, kc[kb].y, qf[kb].x, qf[kb].y);
        mma_16816<T>(s1, ka[kb].z, kc[kb].z, ka[kb].w, kc[kb].w, qf[kb].z, qf[kb].w);
      }
      // s[0], s[1]: token r, heads 2j, 2j + 1;  s[2], s[3]: token r + 8
      float p[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // matmul output rounded to the model dtype, then "/ sqrt(head_dim)" (modeling_gemma.py:266); a power-of-two divisor is
        // applied as an exact multiply
        const float sr = rnd<T>(s0[e] + s1[e]);
        const float sc = (scale_mul != 0.f) ? sr * scale_mul : rnd<T>(sr / scale_div);
        p[e] = (e < 2 ? r : r + 8) <= last ? sc : -INFINITY;
      }
      float corr[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float mx = fmaxf(p[h], p[h + 2]);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float mn = fmaxf(m[h], mx), ref = mn == -INFINITY ? 0.f : mn;   // -inf: no key so far has any weight
        corr[h] = __expf(m[h] - ref);
        m[h] = mn;
        p[h] = __expf(p[h] - ref);
        p[h + 2] = __expf(p[h + 2] - ref);
        l[h] = l[h] * corr[h] + (p[h] + p[h + 2]);              // this lane's tokens; the lanes meet at the end
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) p[e] *= split_scale<T>();
      if constexpr (!fp32) add_values<T, VB>(acc, va, p, corr);
      else add_values_fp32<T, VB, ROPE>(acc, [&](int k) { return vp + k * row_elems; }, p, corr, last + 1);
    }
  };
  attend(std::false_type{});
  if (any_nan(acc)) attend(std::true_type{});                 // an infinity among the values: once more
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);

  // ---- merge the warps of this CTA (those that met a chunk) and hand the sums to the CTAs that finish them.  A CTA writes into its
  // peers' shared memory and reads only its own: fetched from the peers the sums were 48 loads a thread behind the barrier, and a
  // second barrier kept everybody until the last one had read.  The weights of a merge are computed once, a lane each, and go
  // round by shuffle; computed anew for every output they were 4 and 16 exponentials a thread.
  const int busy = min(DM_WARPS, (max(0, chunks - rank) + NS - 1) / NS), per = G * DM_HD / NS;
  auto push4 = [&](int e, const float4& v) {                  // outputs e .. e + 3 of this CTA
    const int to = e / per;
    *reinterpret_cast<float4*>(cluster.map_shared_rank(r_acc + rank * per + (e - to * per), to)) = v;
  };
  auto push_ml = [&](int t, float m_g, float l_g) {           // t: receiving CTA and head
    *cluster.map_shared_rank(&r_ml[rank][t % G], t / G) = make_float2(m_g, l_g);
  };
  if (busy > 1 && wid < busy) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (r == 0) { s_m[wid][2 * j + h] = m[h]; s_l[wid][2 * j + h] = l[h]; }
#pragma unroll
      for (int vb = 0; vb < VB; ++vb) {
        store_acc<T>(&s_acc[wid][2 * j + h][vb * 64 + r * 8], acc[vb], h);
      }
    }
  }
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");             // every CTA of the cluster is there
  if (busy == 1) {                                            // one warp met a chunk: its sums are the CTA's
    if (wid == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int g = 2 * j + h;
        if (g < G) {
#pragma unroll
          for (int vb = 0; vb < VB; ++vb) {
            float v[8];
            store_acc<T>(v, acc[vb], h);
            push4(g * DM_HD + vb * 64 + r * 8, make_float4(v[0], v[1], v[2], v[3]));
            push4(g * DM_HD + vb * 64 + r * 8 + 4, make_float4(v[4], v[5], v[6], v[7]));
          }
          for (int to = r; to < NS; to += 8) push_ml(to * G + g, m[h], l[h]);
        }
      }
    }
  } else if (busy > 1) {
    __syncthreads();
    for (int g = wid; g < G; g += DM_WARPS) {                 // a warp per head, its lanes' weights by shuffle
      float mw = lane < busy ? s_m[lane & (DM_WARPS - 1)][g] : -INFINITY, lw = s_l[lane & (DM_WARPS - 1)][g], M = mw;
#pragma unroll
      for (int o = 1; o < DM_WARPS; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
      M = __shfl_sync(0xffffffffu, M, 0);
      const float fw = mw == -INFINITY ? 0.f : __expf(mw - M);             // a warp whose tokens have no weight
      float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
      float L = 0.f;
#pragma unroll
      for (int w = 0; w < DM_WARPS; ++w) {
        if (w >= busy || __shfl_sync(0xffffffffu, mw, w) == -INFINITY) continue;
        const float f = __shfl_sync(0xffffffffu, fw, w);
        const float4 u = *reinterpret_cast<const float4*>(&s_acc[w][g][lane * 4]);
        const float4 v = *reinterpret_cast<const float4*>(&s_acc[w][g][128 + lane * 4]);
        L = fmaf(f, __shfl_sync(0xffffffffu, lw, w), L);
        a0.x = fmaf(f, u.x, a0.x); a0.y = fmaf(f, u.y, a0.y); a0.z = fmaf(f, u.z, a0.z); a0.w = fmaf(f, u.w, a0.w);
        a1.x = fmaf(f, v.x, a1.x); a1.y = fmaf(f, v.y, a1.y); a1.z = fmaf(f, v.z, a1.z); a1.w = fmaf(f, v.w, a1.w);
      }
      push4(g * DM_HD + lane * 4, a0);
      push4(g * DM_HD + 128 + lane * 4, a1);
      if (lane < NS) push_ml(lane * G + g, M, L);
    }
  }
  __syncwarp();
  cluster.sync();  // what was handed over is there; from here on a CTA reads its own shared memory only

  // ---- this CTA's share of the G * 256 outputs, from the CTAs that met a chunk
  const int n_cta = min(NS, chunks);
  for (int e0 = wid * 32; e0 < per; e0 += DM_WARPS * 32) {    // per is a multiple of 16: half a warp has one head
    const int e = e0 + lane, i = lane & 15, g = min((rank * per + e) / DM_HD, G - 1), d = (rank * per + e) % DM_HD;
    const float2 ml = i < n_cta ? r_ml[i & (NS - 1)][g] : make_float2(-INFINITY, 0.f);   // lane i: CTA i's
    float M = ml.x;
#pragma unroll
    for (int o = 1; o < NS; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o, 16));
    const float wi = ml.x == -INFINITY ? 0.f : __expf(ml.x - M);
    float a = 0.f, L = 0.f;
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      const float mc = __shfl_sync(0xffffffffu, ml.x, c, 16), w = __shfl_sync(0xffffffffu, wi, c, 16);
      const float lc = __shfl_sync(0xffffffffu, ml.y, c, 16);
      if (mc != -INFINITY && e < per) {
        a = fmaf(w, r_acc[c * per + e], a);
        L = fmaf(w, lc, L);
      }
    }
    if (e < per)
      out[((size_t)b * nq + (size_t)kvh * G + g) * DM_HD + d] = from_f<T>(a / L);
  }
}

template <typename T, int NS, bool ROPE, bool AHEAD>
static int launch_dm(void* out, const void* q, const void* k_pool, const void* v_pool, const int32_t* page_table, int pt_stride,
                     int page_size, int num_pages, const int32_t* kv_len, int kv_len_add, int B, int nq, int nkv, float scale_div,
                     const DecodeRope& rope, Prefetch pf, cudaStream_t st) {
  auto kern = decode_attention_mma_kernel<T, NS, ROPE, AHEAD>;
  if (NS > 8) cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(NS, B, nkv);
  cfg.blockDim = dim3(DM_WARPS * 32);
  cfg.stream = st;
  static const int pdl = env_int("PG_PDL", 1);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = NS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (T*)out, (const T*)q, (const T*)k_pool, (const T*)v_pool, page_table, pt_stride,
                                     page_size, num_pages, kv_len, kv_len_add, nq, nkv, scale_div, exact_reciprocal(scale_div), rope, pf);
  if (e != cudaSuccess) {
    set_error("decode_attention launch: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  return check_launch("decode_attention");
}

template <typename T, bool ROPE, bool AHEAD>
static int launch_dm_ns(void* out, const void* q, const void* k_pool, const void* v_pool, const int32_t* page_table, int pt_stride,
                        int page_size, int num_pages, const int32_t* kv_len, int kv_len_add, int B, int nq, int nkv, float scale_div,
                        Prefetch pf, cudaStream_t st, const DecodeRope& rope) {
  // As many CTAs per (sequence, kv head) as keep the launch within one wave of two per SM (16 is a non-portable size), as far as
  // the GPCs have room for whole clusters: 14 of 16, 33 of 8, 70 of 4.  One cluster more takes a second wave
  // (262 cached tokens: 14 sequences 8.9 us, 15 with clusters of 16 14.3).
  const int seqs = B * nkv;
#define PG_DM(N_) \
  return launch_dm<T, N_, ROPE, AHEAD>(out, q, k_pool, v_pool, page_table, pt_stride, page_size, num_pages, kv_len, kv_len_add, B, nq, nkv, \
                                scale_div, rope, pf, st)
  if (seqs <= 14) PG_DM(16);
  if (seqs <= 33) PG_DM(8);
  if (seqs <= 70) PG_DM(4);
  if (seqs <= 148) PG_DM(2);
  PG_DM(1);
#undef PG_DM
}

}  // namespace pg

using namespace pg;

// the mma kernel: 16-bit pools of 256-wide heads in 16-byte aligned rows, whole 16-token chunks inside a page, and query
// heads that fit its 8 columns; everything else (fp32, other head sizes) stays on the general kernel
static bool decode_mma_wanted(const void* q, const void* k_pool, const void* v_pool, int page_size, int G, int hd) {
  const bool aligned = (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0;
  return hd == DM_HD && (G == 1 || G == 2 || G == 4 || G == DM_G) && page_size > 0 && page_size % 16 == 0 && aligned;
}

extern "C" {

int pg_rope_append(void* q_out, const void* qkv, const float* inv_freq, const int32_t* positions, void* k_pool, void* v_pool,
                   const int32_t* page_table, int pt_stride, int page_size, const int32_t* slot_base, int B, int q_len, int nq,
                   int nkv, int hd, int max_pos, int dtype, void* stream);
// One token of each sequence.  qkv: the q/k/v projections, rotated and appended first, in the same launch where the mma kernel takes
// them, else by pg_rope_append into `q` (room for the rotated queries); NULL: q is rotated already and the row in the cache.
int pg_decode_attention_ex(void* out, void* q, void* k_pool, void* v_pool, const int32_t* page_table, int pt_stride, int page_size,
                           int num_pages, const int32_t* kv_len, int kv_len_add, int B, int nq, int nkv, int hd, float scale_div,
                           const void* qkv, const float* inv_freq, const int32_t* positions, int max_pos, int dtype, void* stream) {
  const Prefetch pf = take_prefetch();
  PG_REQUIRE(B > 0 && B <= 65535 && nkv > 0 && nq % nkv == 0, "decode_attention: bad shape");
  PG_REQUIRE(!qkv || kv_len_add == 1, "decode_attention: the appended row is one more than kv_len");
  const int G = nq / nkv;
  cudaStream_t st = (cudaStream_t)stream;
  const void* rows = qkv ? qkv : q;
  if (decode_mma_wanted(rows, k_pool, v_pool, page_size, G, hd) && (!qkv || ((uintptr_t)inv_freq & 7) == 0) &&
      (dtype == PG_BF16 || dtype == PG_F16)) {
    const DecodeRope rope{inv_freq, positions, max_pos};
#define PG_DM(ROPE, AHEAD)                                                                                                       \
  return (dtype == PG_BF16 ? launch_dm_ns<bf16, ROPE, AHEAD> : launch_dm_ns<f16, ROPE, AHEAD>)(                                    \
      out, rows, k_pool, v_pool, page_table, pt_stride, page_size, num_pages, kv_len, kv_len_add, B, nq, nkv, scale_div, pf, st, rope)
    if (qkv) PG_DM(true, true);       // not counted: its pages are all past the end
    if (num_pages > 0) PG_DM(false, true);
    PG_DM(false, false);
#undef PG_DM
  }
  if (qkv) {
    const int rc = pg_rope_append(q, qkv, inv_freq, positions, k_pool, v_pool, page_table, pt_stride, page_size, kv_len, B, 1, nq, nkv,
                                  hd, max_pos, dtype, stream);
    if (rc != PG_OK) return rc;
  }
#define PG_DA(GG, NCH) \
  return launch_da<T, GG, NCH>(out, q, k_pool, v_pool, page_table, pt_stride, page_size, kv_len, kv_len_add, B, nq, nkv, hd, scale_div, pf, st)
  PG_DISPATCH_DTYPE(dtype, T, {
    constexpr int V = Vec<T>::N;
    PG_REQUIRE(hd % V == 0 && hd % 4 == 0 && hd <= 64 * V, "decode_attention: unsupported head_dim %d", hd);
    const int nch = (hd + 32 * V - 1) / (32 * V);
    if (nch == 1) {
      switch (G) {
        case 1: PG_DA(1, 1);
        case 2: PG_DA(2, 1);
        case 4: PG_DA(4, 1);
        case 8: PG_DA(8, 1);
        default: set_error("decode_attention: unsupported group size %d", G); return PG_ERR_INVALID;
      }
    } else {
      switch (G) {
        case 1: PG_DA(1, 2);
        case 2: PG_DA(2, 2);
        case 4: PG_DA(4, 2);
        case 8: PG_DA(8, 2);
        default: set_error("decode_attention: unsupported group size %d", G); return PG_ERR_INVALID;
      }
    }
  });
#undef PG_DA
  return PG_OK;
}

int pg_decode_attention(void* out, const void* q, const void* k_pool, const void* v_pool, const int32_t* page_table, int pt_stride,
                        int page_size, const int32_t* kv_len, int kv_len_add, int B, int nq, int nkv, int hd, float scale_div,
                        float* /*ws*/, int* /*counters*/, int /*max_splits*/, int dtype, void* stream) {
  return pg_decode_attention_ex(out, const_cast<void*>(q), const_cast<void*>(k_pool), const_cast<void*>(v_pool), page_table, pt_stride,
                                page_size, 0, kv_len, kv_len_add, B, nq, nkv, hd, scale_div, nullptr, nullptr, nullptr, 0, dtype, stream);
}

int pg_decode_attention_rope(void* out, void* q, const void* qkv, const float* inv_freq, const int32_t* positions, void* k_pool,
                             void* v_pool, const int32_t* page_table, int pt_stride, int page_size, const int32_t* kv_len, int B,
                             int nq, int nkv, int hd, int max_pos, float scale_div, int dtype, void* stream) {
  PG_REQUIRE(qkv, "decode_attention_rope: no projections");
  return pg_decode_attention_ex(out, q, k_pool, v_pool, page_table, pt_stride, page_size, 0, kv_len, 1, B, nq, nkv, hd, scale_div, qkv,
                                inv_freq, positions, max_pos, dtype, stream);
}

long long pg_decode_attention_ws_floats(int, int, int, int) { return 0; }

}  // extern "C"
