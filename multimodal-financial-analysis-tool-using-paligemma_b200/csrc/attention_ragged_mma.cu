// Attention of single tokens over the paged cache on mma.sync (16-bit types): the decode-sized steps of attention_ragged.cu,
// same masks, weights and epilogue.
//
// One thread-block cluster per (token, key/value head, up to 8 of its query heads); the cluster's warps take the visible keys 16
// at a time, chunk c by CTA c % CTAs, warp c / CTAs.  With the query heads as the N dimension of mma.m16n8k16
//   S^T [16 keys x 8 heads] = K Q^T,   O^T [vdim x 8 heads] += V^T P^T
// every key and value row is read once for the whole group, straight into fragments with 16-byte loads: the contraction index of
// S^T is permuted (lane j of a quad owns 8 consecutive columns of every 32), and so are the rows of O^T (lane group r owns 8
// consecutive columns of every 64).  Q K^T multiplies the stored 16-bit operands; the weights stay fp32 and enter P V as three
// 16-bit terms (mma_frag.cuh): all their 24 bits in bf16, 2^-39 of the largest weight in fp16; fp16 sigmoid weights, which no
// maximum normalises, stay with the fp32 kernels.  (m, l, O) of the warps meet in shared memory and those of the CTAs in
// distributed shared memory, in a fixed order: one launch, no workspace.
// The key-slice kernel of attention_ragged.cu gives a whole key row to one lane (32 rows of 16 bytes per load), keeps the query
// in shared memory and needs a second launch to merge: 8 tokens x 1024 keys, 16 heads over 4, 128 wide: 30.2 + 9.7 us, this
// kernel 13.7 us (launch alone, cold cache; 31.9 -> 9.6 us in a row of steps), the bytes alone 2.6 us: what is left is the chain
// token -> page -> rows -> merge.
#include <cooperative_groups.h>

#include "attention_ragged.cuh"
#include "mma_frag.cuh"

namespace cg = cooperative_groups;

namespace pg {

constexpr int RM_WARPS = 4, RM_G = 8, RM_MAX_CTAS = 16;

template <typename T, int KB, int VB>    // key width 32 KB, value width 64 VB
__global__ void __launch_bounds__(RM_WARPS * 32, 2)
attention_ragged_mma_kernel(RagAttnParams p, int head_chunks) {
  constexpr int DIM = 32 * KB, VDIM = 64 * VB;
  cg::cluster_group cluster = cg::this_cluster();
  const int ns = (int)gridDim.x, rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, r = lane >> 2, j = lane & 3;
  const int per_tok = p.G * head_chunks, t = blockIdx.y / per_tok, gc = blockIdx.y % per_tok, g = gc / head_chunks;
  const int group = p.H / p.G, first = (gc % head_chunks) * RM_G, h0 = g * group + first, hn = min(RM_G, group - first);
  __shared__ __align__(16) float s_acc[RM_WARPS][RM_G][VDIM];
  __shared__ __align__(16) float c_acc[RM_G][VDIM];       // CTA-level partial (read by peers)
  __shared__ float s_m[RM_WARPS][RM_G], s_l[RM_WARPS][RM_G], c_m[RM_G], c_l[RM_G];
  pdl_launch_dependents();
  pdl_wait();
  const int pos = p.tok_pos[t];
  const int32_t* pt_row = p.page_table + (size_t)p.tok_slot[t] * p.pt_stride;
  uint4 qf[KB];
  {
    const T* qr = reinterpret_cast<const T*>(p.q) + (size_t)t * p.ld_q + (size_t)(h0 + r) * DIM + j * 8;
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) qf[kb] = r < hn ? ldg_cached(qr + kb * 32) : make_uint4(0, 0, 0, 0);
  }
  float slope[2], bias[2];                                // heads 2j and 2j + 1
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int hh = h0 + min(2 * j + h, hn - 1);
    slope[h] = p.slopes ? p.slopes[hh] : 0.f;
    bias[h] = p.head_bias ? p.head_bias[hh] : 0.f;
  }
  const KeyRange kr(pos, p.window, p.keep_first, p.chunk);
  const float qscale = query_scale(p, pos);
  const T* kpool = reinterpret_cast<const T*>(p.k_pool) + (size_t)g * DIM + j * 8;
  const T* vpool = reinterpret_cast<const T*>(p.v_pool) + (size_t)g * VDIM + r * 8;
  const float m_init = p.sigmoid_weights ? 0.f : -INFINITY;
  float acc[VB][4][4], m[2], l[2];                        // m, l: the same in every lane group

  const int chunks = (kr.count + 15) / 16, stride = ns * RM_WARPS;
  // lane L looks up key L % 16 of a chunk (positions behind the last key repeat it, with weight 0): its position and pool row
  int key = 0, row = 0;
  auto look_up = [&](int c) {
    key = kr.key(min(16 * c + (lane & 15), kr.count - 1));
    row = pt_row[key / p.page_size] * p.page_size + key % p.page_size;
  };
  for (bool in_fp32 = false;; in_fp32 = true) {
#pragma unroll
  for (int vb = 0; vb < VB; ++vb)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[vb][i][e] = 0.f;
  m[0] = m[1] = m_init;
  l[0] = l[1] = 0.f;
  int c = rank + ns * wid;
  if (c < chunks) look_up(c);
  for (; c < chunks; c += stride) {
    const int n = kr.count - 16 * c;                       // keys of this chunk (16 and more: all)
    const int key0 = __shfl_sync(0xffffffffu, key, r), key1 = __shfl_sync(0xffffffffu, key, r + 8);
    const size_t k0 = (size_t)__shfl_sync(0xffffffffu, row, r) * p.ld_k, k1 = (size_t)__shfl_sync(0xffffffffu, row, r + 8) * p.ld_k;
    const size_t v0 = (size_t)__shfl_sync(0xffffffffu, row, 2 * j) * p.ld_v, v1 = (size_t)__shfl_sync(0xffffffffu, row, 2 * j + 1) * p.ld_v;
    const size_t v2 = (size_t)__shfl_sync(0xffffffffu, row, 2 * j + 8) * p.ld_v, v3 = (size_t)__shfl_sync(0xffffffffu, row, 2 * j + 9) * p.ld_v;
    uint4 ka[KB], kc[KB], va[VB][4];
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) { ka[kb] = ldg_cached(kpool + k0 + kb * 32); kc[kb] = ldg_cached(kpool + k1 + kb * 32); }
#pragma unroll
    for (int vb = 0; vb < VB; ++vb) {
      va[vb][0] = ldg_cached(vpool + v0 + vb * 64); va[vb][1] = ldg_cached(vpool + v1 + vb * 64);
      va[vb][2] = ldg_cached(vpool + v2 + vb * 64); va[vb][3] = ldg_cached(vpool + v3 + vb * 64);
    }
    if (!in_fp32 && c + stride < chunks) look_up(c + stride);   // the next chunk's pages come in beside this one's rows
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
      mma_16816<T>(s0, ka[kb].x, kc[kb].x, ka[kb].y, kc[kb].y, qf[kb].x, qf[kb].y);
      mma_16816<T>(s1, ka[kb].z, kc[kb].z, ka[kb].w, kc[kb].w, qf[kb].z, qf[kb].w);
    }
    // w[0], w[1]: key r, heads 2j, 2j + 1;  w[2], w[3]: key r + 8
    float w[4], corr[2] = {1.f, 1.f};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float sc = capped(p, (s0[e] + s1[e]) * qscale) - slope[e & 1] * (float)(pos - (e < 2 ? key0 : key1)) + bias[e & 1];
      w[e] = (e < 2 ? r : r + 8) < n ? sc : -INFINITY;
    }
    if (p.sigmoid_weights) {                               // unnormalised: no running maximum
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = w[e] == -INFINITY ? 0.f : 1.f / (1.f + expf(-w[e]));
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float mx = fmaxf(w[h], w[h + 2]);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float mn = fmaxf(m[h], mx), ref = mn == -INFINITY ? 0.f : mn;   // -inf: no key so far has any weight
        corr[h] = expf(m[h] - ref);
        m[h] = mn;
        w[h] = expf(w[h] - ref);
        w[h + 2] = expf(w[h + 2] - ref);
        l[h] = l[h] * corr[h] + (w[h] + w[h + 2]);          // this lane's keys; the lanes meet at the end
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] *= split_scale<T>();
    if (!in_fp32) {
      add_values<T, VB>(acc, va, w, corr);
    } else {
      add_values_fp32<T, VB>(acc, [&](int k) { return vpool + (size_t)__shfl_sync(0xffffffffu, row, k) * p.ld_v; }, w, corr, n);
      if (c + stride < chunks) look_up(c + stride);
    }
  }
  if (in_fp32 || !any_nan(acc)) break;                      // an infinity among the values: once more
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);

  // ---- merge the warps of this CTA (those that met a chunk)
  const int busy = min(RM_WARPS, (max(0, chunks - rank) + ns - 1) / ns);
  if (wid < busy) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (r == 0) { s_m[wid][2 * j + h] = m[h]; s_l[wid][2 * j + h] = l[h]; }
#pragma unroll
      for (int vb = 0; vb < VB; ++vb) {
        store_acc<T>(&s_acc[wid][2 * j + h][vb * 64 + r * 8], acc[vb], h);
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x * 4; e < hn * VDIM; e += RM_WARPS * 32 * 4) {
    const int hh = e / VDIM, d = e % VDIM;
    float M = -INFINITY;
    for (int k = 0; k < busy; ++k) M = fmaxf(M, s_m[k][hh]);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    float L = 0.f;
    for (int k = 0; k < busy; ++k) {
      if (s_m[k][hh] == -INFINITY) continue;                // a warp whose keys have no weight
      const float f = expf(s_m[k][hh] - M);
      const float4 v = *reinterpret_cast<const float4*>(&s_acc[k][hh][d]);
      a.x = fmaf(f, v.x, a.x); a.y = fmaf(f, v.y, a.y); a.z = fmaf(f, v.z, a.z); a.w = fmaf(f, v.w, a.w);
      L = fmaf(f, s_l[k][hh], L);
    }
    *reinterpret_cast<float4*>(&c_acc[hh][d]) = a;
    if (d == 0) { c_m[hh] = M; c_l[hh] = L; }
  }
  cluster.sync();  // every CTA's partial is visible cluster-wide

  // ---- merge the CTAs that met a chunk: CTA `rank` finishes its slice of the hn * VDIM outputs
  const int n_cta = min(ns, chunks);
  auto merged = [&](int hh, int d) {
    float pm[RM_MAX_CTAS], pl[RM_MAX_CTAS], pa[RM_MAX_CTAS];
#pragma unroll
    for (int i = 0; i < RM_MAX_CTAS; ++i) {
      const bool have = i < n_cta;
      pm[i] = have ? *cluster.map_shared_rank(&c_m[hh], i) : -INFINITY;
      pl[i] = have ? *cluster.map_shared_rank(&c_l[hh], i) : 0.f;
      pa[i] = have ? *cluster.map_shared_rank(&c_acc[hh][d], i) : 0.f;
    }
    float M = -INFINITY;
#pragma unroll
    for (int i = 0; i < RM_MAX_CTAS; ++i) M = fmaxf(M, pm[i]);
    float a = 0.f, L = 0.f;
#pragma unroll
    for (int i = 0; i < RM_MAX_CTAS; ++i)
      if (i < n_cta && pm[i] != -INFINITY) {
        const float f = expf(pm[i] - M);
        a = fmaf(f, pa[i], a);
        L = fmaf(f, pl[i], L);
      }
    if (p.sigmoid_weights) return a;
    if (p.sink) L += expf(p.sink[h0 + hh] - M);            // a logit without key or value, counted once
    return a / L;
  };
  const int per = (hn * VDIM + ns - 1) / ns, e_end = min(hn * VDIM, (rank + 1) * per);
  for (int e = rank * per + threadIdx.x; e < e_end; e += RM_WARPS * 32) {
    const int hh = e / VDIM, d = e % VDIM, h = h0 + hh;
    float v = merged(hh, d);
    if (p.out_rot) {                                       // turned back by the query's position, before the gate
      const int half = VDIM / 2;
      const bool lo = p.out_rot_interleaved ? !(d & 1) : d < half;
      const int pair = p.out_rot_interleaved ? d >> 1 : (lo ? d : d - half);
      const float other = merged(hh, p.out_rot_interleaved ? d ^ 1 : (lo ? d + half : d - half));
      float sn, cs;
      sincosf(-(float)pos * p.out_rot[pair], &sn, &cs);
      v = lo ? v * cs - other * sn : v * cs + other * sn;
    }
    v *= p.out_scale;
    if (p.gate) {
      const T* gt = reinterpret_cast<const T*>(p.gate) + (size_t)t * p.ld_gate;
      v *= 1.f / (1.f + expf(-to_f<T>(p.gate_per_head ? gt[h] : gt[(size_t)h * VDIM + d])));
    }
    reinterpret_cast<T*>(p.out)[(size_t)t * p.ld_out + (size_t)h * VDIM + d] = from_f<T>(v);
  }
  cluster.sync();  // nobody leaves while a peer may still read its shared memory
}

template <typename T, int KB, int VB>
static int launch_rm(const RagAttnParams& p, cudaStream_t st) {
  auto kern = attention_ragged_mma_kernel<T, KB, VB>;
  const int head_chunks = cdiv(p.H / p.G, RM_G);
  const long long groups = (long long)p.n_tokens * p.G * head_chunks;
  // CTAs per group of heads: until two per SM are busy, as long as a warp keeps two chunks of 16 keys (16 is a non-portable size)
  int span = p.window > 0 ? p.window + max(p.keep_first, 0) : 1 << 20, ns = 1;
  if (p.chunk > 0) span = min(span, p.chunk);
  while (ns < RM_MAX_CTAS && groups * ns * 2 <= 296 && span / (ns * 2) >= 32 * RM_WARPS) ns *= 2;
  cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ns, (unsigned)groups);
  cfg.blockDim = dim3(RM_WARPS * 32);
  cfg.stream = st;
  static const int pdl = env_int("PG_PDL", 1);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ns;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, head_chunks);
  if (e != cudaSuccess) {
    set_error("attention_ragged_mma launch: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  return check_launch("attention_ragged_mma");
}

// (key width, value width) pairs the kernel is built for, weights its 16-bit terms hold (mma_frag.cuh); everything it loads in
// 16 bytes lies on 16-byte boundaries
bool attention_ragged_mma_wanted(const RagAttnParams& p, int dtype) {
  if (dtype != PG_BF16 && (dtype != PG_F16 || p.sigmoid_weights)) return false;
  const bool square = p.dim == p.vdim && (p.dim == 64 || p.dim == 128 || p.dim == 256);
  if (!square && !(p.dim == 256 && p.vdim == 192)) return false;
  if (p.ld_q % 8 || p.ld_k % 8 || p.ld_v % 8 || (((uintptr_t)p.q | (uintptr_t)p.k_pool | (uintptr_t)p.v_pool) & 15)) return false;
  return (long long)p.n_tokens * p.G * cdiv(p.H / p.G, RM_G) <= 65535;
}

template <typename T>
static int launch_rm_any(const RagAttnParams& p, cudaStream_t st) {
  if (p.dim == 64) return launch_rm<T, 2, 1>(p, st);
  if (p.dim == 128) return launch_rm<T, 4, 2>(p, st);
  return p.vdim == 192 ? launch_rm<T, 8, 3>(p, st) : launch_rm<T, 8, 4>(p, st);
}

int attention_ragged_mma(const RagAttnParams& p, int dtype, cudaStream_t st) {
  return dtype == PG_BF16 ? launch_rm_any<bf16>(p, st) : launch_rm_any<f16>(p, st);
}

}  // namespace pg
