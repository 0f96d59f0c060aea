// Row / elementwise kernels of the PaliGemma path: embedding+merge, norms, im2col, RoPE+KV
// append (prefill), step bookkeeping, argmax, KV gather.  All HBM-bound; 128-bit accesses.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <atomic>

#include "common.cuh"
#include "tp_exchange.cuh"

namespace pg {

static thread_local char g_err[512] = "";
static std::atomic<unsigned long long> g_launches{0};
static thread_local Prefetch g_prefetch = {nullptr, 0};

int env_int(const char* name, int dflt) {
  const char* v = getenv(name);
  return (v && *v) ? atoi(v) : dflt;
}

Prefetch take_prefetch() {
  Prefetch p = g_prefetch;
  g_prefetch = {nullptr, 0};
  return p;
}

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int check_launch(const char* what) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  cudaError_t e = cudaPeekAtLastError();
  if (e != cudaSuccess) {
    set_error("%s: %s", what, cudaGetErrorString(e));
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  return PG_OK;
}

// ------------------------------------------------------------------ embed + merge
// One CTA per token.  The k-th image token (row-major over the flattened ids) takes image row k
// (masked_scatter order, modeling_gemma.py:498).  The first token that is an error is described in info (id, t, the step's
// number or -1) before the flag is set.
template <typename T>
__global__ void embed_merge_kernel(T* __restrict__ out, const int64_t* __restrict__ ids,
                                   const T* __restrict__ emb, const T* __restrict__ img,
                                   int n_tokens, int D, int64_t vocab, int64_t img_id, int64_t pad_id,
                                   int n_img_rows, float img_div, float normalizer, int* err_flag, int drawn,
                                   const int32_t* __restrict__ step, long long* info) {
  pdl_launch_dependents();  // a tensor-core kernel launched next may start its prologue now
  constexpr int V = Vec<T>::N;
  __shared__ float red[32];
  const int t = blockIdx.x;
  const int64_t id = ids[t];
  const T* src = nullptr;
  bool is_img = false, bad = false;
  if (id == img_id) {
    float cnt = 0.f;
    for (int i = threadIdx.x; i < t; i += blockDim.x) cnt += (ids[i] == img_id) ? 1.f : 0.f;
    int k = (int)(block_sum(cnt, red) + 0.5f);
    if (img != nullptr && k < n_img_rows) { src = img + (size_t)k * D; is_img = true; }
    else bad = drawn == 0;
  } else if (id != pad_id) {
    if (id >= 0 && id < vocab) src = emb + (size_t)id * D;
    else bad = true;
  }
  if (bad && err_flag) {                                 // rare: is an earlier token the one to name?
    float outside = 0.f, images = 0.f;
    for (int i = threadIdx.x; i < t; i += blockDim.x) {
      const int64_t x = ids[i];
      if (x == img_id) images += 1.f;
      else if (x != pad_id && (x < 0 || x >= vocab)) outside += 1.f;
    }
    outside = block_sum(outside, red);
    images = drawn ? 0.f : block_sum(images, red);
    const int rows = img != nullptr ? n_img_rows : 0;
    if (threadIdx.x == 0 && outside == 0.f && images <= (float)rows) {
      if (info && *(volatile int*)err_flag == 0) {
        info[0] = id;
        info[1] = t;
        info[2] = step ? *step : -1;
        __threadfence_system();
      }
      *(volatile int*)err_flag = 1;
    }
  }
  T* dst = out + (size_t)t * D;
  for (int c = threadIdx.x * V; c < D; c += blockDim.x * V) {
    float f[V];
    if (src) {
      unpack<T>(ldg_cached(src + c), f);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float v = f[i];
        if (is_img) v = rnd<T>(v / img_div);
        f[i] = v * normalizer;
      }
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) f[i] = 0.f;
    }
    *reinterpret_cast<uint4*>(dst + c) = pack<T>(f);
  }
}

// ------------------------------------------------------------------ RMSNorm / LayerNorm
// One CTA per row; the row is kept in registers between the statistics pass and the write.
template <typename T, int MAXV>
__global__ void rmsnorm_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ w,
                               int D, float eps) {
  pdl_launch_dependents();  // a tensor-core kernel launched next may start its prologue now
  pdl_wait();               // (launched with the PDL attribute when the grid is small: inputs come from the predecessor)
  constexpr int V = Vec<T>::N;
  __shared__ float red[32];
  const T* xr = x + (size_t)blockIdx.x * D;
  T* orow = out + (size_t)blockIdx.x * D;
  float f[MAXV][V];
  uint4 wr[MAXV];             // the weights come in beside the row: behind the reduction they were a second trip to HBM
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    int c = (j * blockDim.x + threadIdx.x) * V;
    wr[j] = c < D ? ldg_cached(w + c) : make_uint4(0, 0, 0, 0);
    if (c < D) {
      unpack<T>(ldg_cached(xr + c), f[j]);
#pragma unroll
      for (int i = 0; i < V; ++i) ss += f[j][i] * f[j][i];
    }
  }
  ss = block_sum(ss, red);
  const float inv = rsqrtf(ss / (float)D + eps);
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    int c = (j * blockDim.x + threadIdx.x) * V;
    if (c < D) {
      float g[V];
      unpack<T>(wr[j], g);
#pragma unroll
      for (int i = 0; i < V; ++i) f[j][i] = (f[j][i] * inv) * (1.0f + g[i]);
      *reinterpret_cast<uint4*>(orow + c) = pack<T>(f[j]);
    }
  }
}

template <typename T, int MAXV>
__global__ void layernorm_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ w,
                                 const T* __restrict__ b, int D, float eps) {
  pdl_launch_dependents();  // a tensor-core kernel launched next may start its prologue now
  pdl_wait();               // (launched with the PDL attribute when the grid is small: inputs come from the predecessor)
  constexpr int V = Vec<T>::N;
  __shared__ float red[32];
  const T* xr = x + (size_t)blockIdx.x * D;
  T* orow = out + (size_t)blockIdx.x * D;
  float f[MAXV][V];
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    int c = (j * blockDim.x + threadIdx.x) * V;
    if (c < D) {
      unpack<T>(ldg_cached(xr + c), f[j]);
#pragma unroll
      for (int i = 0; i < V; ++i) s += f[j][i];
    }
  }
  const float mean = block_sum(s, red) / (float)D;
  float q = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    int c = (j * blockDim.x + threadIdx.x) * V;
    if (c < D) {
#pragma unroll
      for (int i = 0; i < V; ++i) { float d = f[j][i] - mean; q += d * d; }
    }
  }
  const float rstd = rsqrtf(block_sum(q, red) / (float)D + eps);
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    int c = (j * blockDim.x + threadIdx.x) * V;
    if (c < D) {
      float g[V], bb[V];
      unpack<T>(ldg_cached(w + c), g);
      unpack<T>(ldg_cached(b + c), bb);
#pragma unroll
      for (int i = 0; i < V; ++i) f[j][i] = (f[j][i] - mean) * rstd * g[i] + bb[i];
      *reinterpret_cast<uint4*>(orow + c) = pack<T>(f[j]);
    }
  }
}


// ------------------------------------------------------------------ warp-per-row norms (many rows)
// Prefill / vision: thousands of rows of 1152-2048 elements.  One warp per row (8 rows per CTA), the row
// stays in registers between the statistics and the write, fully coalesced 16-byte accesses.
// EARLY (up to 1024 rows): the weights are requested together with the row instead of behind the statistics, which are
// then the only thing between the loads and the stores; with thousands of rows the registers are worth more as rows in flight.
// Two rows per CTA there, so that 256 rows reach 128 SMs instead of 32.  One image's encode (19 of these among 66 launches) 575 ->
// 544 us, a 260-token prompt with its image 4855 -> 4674 us.
template <typename T, int MAXV, bool LAYERNORM, bool EARLY>
__global__ void __launch_bounds__(256)
norm_rows_warp_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ b,
                      int rows, int D, float eps) {
  pdl_launch_dependents();  // a tensor-core kernel launched next may start its prologue now
  pdl_wait();               // (launched with the PDL attribute when the grid is small: inputs come from the predecessor)
  constexpr int V = Vec<T>::N;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const T* xr = x + (size_t)row * D;
  T* orow = out + (size_t)row * D;
  // the row is held as the raw 16-byte vectors (4 registers each, unpacked on the fly in every pass): ~45 registers,
  // so 5-6 CTAs (40+ rows) per SM keep enough bytes in flight for HBM
  uint4 raw[MAXV];
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    const int c = (j * 32 + lane) * V;
    raw[j] = c < D ? ldg_cached(xr + c) : make_uint4(0, 0, 0, 0);
  }
  uint4 wr[EARLY ? MAXV : 1], br[EARLY && LAYERNORM ? MAXV : 1];
  if constexpr (EARLY) {
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int c = (j * 32 + lane) * V;
      wr[j] = c < D ? ldg_cached(w + c) : make_uint4(0, 0, 0, 0);
      if constexpr (LAYERNORM) br[j] = c < D ? ldg_cached(b + c) : make_uint4(0, 0, 0, 0);
    }
  }
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    float f[V];
    unpack<T>(raw[j], f);   // out-of-row vectors are zeros: they add nothing to either sum
#pragma unroll
    for (int i = 0; i < V; ++i) s += LAYERNORM ? f[i] : f[i] * f[i];
  }
  s = warp_sum(s);
  float mean = 0.f, scale;
  if (LAYERNORM) {
    mean = s / (float)D;
    float q = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int c = (j * 32 + lane) * V;
      if (c < D) {
        float f[V];
        unpack<T>(raw[j], f);
#pragma unroll
        for (int i = 0; i < V; ++i) { const float d = f[i] - mean; q += d * d; }
      }
    }
    scale = rsqrtf(warp_sum(q) / (float)D + eps);
  } else {
    scale = rsqrtf(s / (float)D + eps);
  }
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    const int c = (j * 32 + lane) * V;
    if (c < D) {
      float f[V], g[V], bb[V];
      unpack<T>(raw[j], f);
      unpack<T>(EARLY ? wr[EARLY ? j : 0] : ldg_cached(w + c), g);
      if (LAYERNORM) unpack<T>(EARLY ? br[EARLY && LAYERNORM ? j : 0] : ldg_cached(b + c), bb);
#pragma unroll
      for (int i = 0; i < V; ++i)
        f[i] = LAYERNORM ? (f[i] - mean) * scale * g[i] + bb[i] : (f[i] * scale) * (1.0f + g[i]);
      *reinterpret_cast<uint4*>(orow + c) = pack<T>(f);
    }
  }
}

// ------------------------------------------------------------------ im2col (stride == kernel)
// The same for even patch sizes on pair boundaries: a thread moves one patch row (p pixels of one channel) as pairs, the
// first thread of a token also zeroes the columns behind C * p * p (64 images of 224 x 224: 68 -> 24 us).
template <typename T>
__global__ void __launch_bounds__(256)
im2col_rows_kernel(T* __restrict__ out, const T* __restrict__ px, int C, int H, int W, int p, int ld_out, int n_rows) {
  struct alignas(2 * sizeof(T)) P { T a, b; };
  const int G = W / p, per_tok = C * p;
  for (long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x; at < n_rows; at += (long long)gridDim.x * blockDim.x) {
    const int idx = (int)at;             // rows are counted in 32 bits; the step behind the last one may not fit
    // neighbouring threads take the same row of neighbouring patches: their loads are consecutive
    const int gx = idx % G, k = idx / G, ky = k % p, k2 = k / p, c = k2 % C, k3 = k2 / C, gy = k3 % (H / p), b = k3 / (H / p);
    const P* src = reinterpret_cast<const P*>(px + (((size_t)b * C + c) * H + gy * p + ky) * W + gx * p);
    T* tok = out + ((size_t)b * (H / p) * G + gy * G + gx) * ld_out;
    P* dst = reinterpret_cast<P*>(tok + (c * p + ky) * p);
#pragma unroll 8
    for (int i = 0; i < p / 2; ++i) dst[i] = src[i];
    if (c == 0 && ky == 0)
      for (int i = per_tok * p; i < ld_out; ++i) tok[i] = from_f<T>(0.f);
  }
}

template <typename T>
__global__ void im2col_kernel(T* __restrict__ out, const T* __restrict__ px, int C, int H, int W, int p,
                              int ld_out, long long total) {
  pdl_launch_dependents();  // a tensor-core kernel launched next may start its prologue now
  const int G = W / p, P = (H / p) * G, Kc = C * p * p;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    int col = (int)(i % ld_out);
    long long row = i / ld_out;
    T v = from_f<T>(0.f);
    if (col < Kc) {
      int b = (int)(row / P), pp = (int)(row % P);
      int py = pp / G, pxx = pp % G;
      int c = col / (p * p), r = col % (p * p);
      int ky = r / p, kx = r % p;
      v = px[(((size_t)b * C + c) * H + (py * p + ky)) * W + (pxx * p + kx)];
    }
    out[i] = v;
  }
}

// ------------------------------------------------------------------ RoPE + KV append (prefill)
// One CTA per token.  Thread j < hd/2 handles the rotation pair (j, j+hd/2) of every head.
template <typename T>
__global__ void rope_append_kernel(T* __restrict__ q_out, const T* __restrict__ qkv,
                                   const float* __restrict__ inv_freq, const int32_t* __restrict__ positions,
                                   T* __restrict__ k_pool, T* __restrict__ v_pool,
                                   const int32_t* __restrict__ page_table, int pt_stride, int page_size,
                                   const int32_t* __restrict__ slot_base, int q_len, int nq, int nkv, int hd,
                                   int max_pos) {
  pdl_launch_dependents();  // a tensor-core kernel launched next may start its prologue now
  pdl_wait();               // (launched with the PDL attribute when the grid is small: inputs come from the predecessor)
  const int t = blockIdx.x, b = t / q_len, i = t % q_len;
  const int half = hd / 2;
  int pos = positions[t];
  pos = min(max(pos, 0), max_pos - 1);
  const int slot = slot_base[b] + i;
  const int page = page_table[(size_t)b * pt_stride + slot / page_size];
  const size_t kv_row = ((size_t)page * page_size + (slot % page_size)) * (size_t)(nkv * hd);
  const T* row = qkv + (size_t)t * (nq + 2 * nkv) * hd;
  T* qo = q_out + (size_t)t * nq * hd;
  // a thread owns one rotation index j (cos / sin evaluated once, reused for every head) and every other head
  const int jl = threadIdx.x % (blockDim.x / 2), hg = threadIdx.x / (blockDim.x / 2);
  for (int j = jl; j < half; j += blockDim.x / 2) {
    const float ang = (float)pos * inv_freq[j];
    const float c = rnd<T>(cosf(ang)), s = rnd<T>(sinf(ang));
#pragma unroll 3
    for (int h = hg; h < nq + nkv; h += 2) {
      const float x1 = to_f<T>(row[h * hd + j]), x2 = to_f<T>(row[h * hd + j + half]);
      const float o1 = rnd<T>(rnd<T>(x1 * c) + rnd<T>(-x2 * s));
      const float o2 = rnd<T>(rnd<T>(x2 * c) + rnd<T>(x1 * s));
      if (h < nq) {
        qo[h * hd + j] = from_f<T>(o1);
        qo[h * hd + j + half] = from_f<T>(o2);
      } else {
        const int kh = h - nq;
        k_pool[kv_row + kh * hd + j] = from_f<T>(o1);
        k_pool[kv_row + kh * hd + j + half] = from_f<T>(o2);
      }
    }
  }
  const T* vrow = row + (size_t)(nq + nkv) * hd;
  for (int u = threadIdx.x; u < nkv * hd; u += blockDim.x) v_pool[kv_row + u] = vrow[u];
}

// The same for head sizes that are multiples of 4 and rows on pair boundaries: a thread owns two neighbouring rotation indices and
// moves them as pairs, CTA (token, y) takes the heads [y * heads_per_cta, ..) of [q | k | v].  A few tokens: one head per CTA,
// so that the chain is position -> cache row -> one load -> one store (8 rows of 10 heads: 7.6 -> 4.3 us); many tokens: all
// heads in one CTA, four at a time (1292 rows: 12.3 -> 10.0 us).
template <typename T> struct alignas(2 * sizeof(T)) Pair2 { T a, b; };

template <typename T>
__global__ void __launch_bounds__(256)
rope_append_pair_kernel(T* __restrict__ q_out, const T* __restrict__ qkv, const float* __restrict__ inv_freq,
                        const int32_t* __restrict__ positions, T* __restrict__ k_pool, T* __restrict__ v_pool,
                        const int32_t* __restrict__ page_table, int pt_stride, int page_size,
                        const int32_t* __restrict__ slot_base, int q_len, int nq, int nkv, int hd, int max_pos,
                        int heads_per_cta) {
  typedef Pair2<T> P;
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, b = t / q_len, i = t % q_len;
  const int half = hd / 2, quarter = hd / 4, jp = threadIdx.x % quarter, groups = blockDim.x / quarter;
  const int pos = min(max(positions[t], 0), max_pos - 1);
  const int slot = slot_base[b] + i;
  const float f0 = inv_freq[2 * jp], f1 = inv_freq[2 * jp + 1];
  const int h_begin = blockIdx.y * heads_per_cta, h_end = min(nq + 2 * nkv, h_begin + heads_per_cta);
  const T* row = qkv + (size_t)t * (nq + 2 * nkv) * hd;
  const int page = page_table[(size_t)b * pt_stride + slot / page_size];
  const size_t kv_row = ((size_t)page * page_size + (slot % page_size)) * (size_t)(nkv * hd);
  const float a0 = (float)pos * f0, a1 = (float)pos * f1;
  const float c0 = rnd<T>(cosf(a0)), s0 = rnd<T>(sinf(a0)), c1 = rnd<T>(cosf(a1)), s1 = rnd<T>(sinf(a1));
#pragma unroll 3
  for (int h = h_begin + threadIdx.x / quarter; h < h_end; h += groups) {
    P lo = *reinterpret_cast<const P*>(row + (size_t)h * hd + 2 * jp), hi = *reinterpret_cast<const P*>(row + (size_t)h * hd + half + 2 * jp);
    if (h < nq + nkv) {
      const float x0 = to_f<T>(lo.a), x1 = to_f<T>(lo.b), y0 = to_f<T>(hi.a), y1 = to_f<T>(hi.b);
      lo.a = from_f<T>(rnd<T>(x0 * c0) + rnd<T>(-y0 * s0));
      lo.b = from_f<T>(rnd<T>(x1 * c1) + rnd<T>(-y1 * s1));
      hi.a = from_f<T>(rnd<T>(y0 * c0) + rnd<T>(x0 * s0));
      hi.b = from_f<T>(rnd<T>(y1 * c1) + rnd<T>(x1 * s1));
    }
    T* dst = h < nq ? q_out + (size_t)t * nq * hd + (size_t)h * hd
                    : (h < nq + nkv ? k_pool + kv_row + (size_t)(h - nq) * hd : v_pool + kv_row + (size_t)(h - nq - nkv) * hd);
    *reinterpret_cast<P*>(dst + 2 * jp) = lo;
    *reinterpret_cast<P*>(dst + half + 2 * jp) = hi;
  }
}

// ------------------------------------------------------------------ decode-step bookkeeping
__global__ void step_advance_kernel(int64_t* next_ids, int64_t* history, int hist_stride, int* step_counter,
                                    unsigned long long* keys, const int64_t* sampled, int32_t* kv_len,
                                    int32_t* positions, int B, TpEx ex) {
  const int b = threadIdx.x;
  const int step = step_counter ? *step_counter : 0;
  __syncthreads();
  if (b < B) {
    // tensor parallel + greedy: the winning (value, global index) key over the ranks' vocabulary shards
    int64_t tok = sampled ? sampled[b]
                          : (int64_t)argmax_key_index(ex.peers ? tp_wait_best_key(ex, b) : keys[b]);
    next_ids[b] = tok;
    // ring index: the step counter (also the sampler's RNG offset) keeps counting for the life of the engine
    if (history && hist_stride > 0) history[(size_t)b * hist_stride + (unsigned)step % (unsigned)hist_stride] = tok;
    if (kv_len) kv_len[b] += 1;
    if (positions) positions[b] += 1;
    keys[b] = 0ull;
  }
  if (b == 0 && step_counter) *step_counter = (int)((unsigned)step + 1u);   // wraps like the ring index above
}

// One launch at the head of an API-driven decode step: token ids and positions into the graph's static buffers,
// plus the reference's all-ones attention-mask check (modeling_gemma.py:559) reported through a flag instead of a
// host synchronisation.
template <typename M>
__device__ __forceinline__ bool mask_is_one(const void* mask, long long i) {
  return reinterpret_cast<const M*>(mask)[i] == (M)1;
}
__global__ void decode_inputs_kernel(int64_t* ids_dst, const int64_t* ids_src, int32_t* positions, int position,
                                     const void* mask, int mask_kind, long long mask_n, int* bad_flag, int B) {
  if (blockIdx.x == 0)
    for (int b = threadIdx.x; b < B; b += blockDim.x) {
      ids_dst[b] = ids_src[b];
      positions[b] = position;
    }
  bool bad = false;
#pragma unroll 4
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < mask_n; i += (long long)gridDim.x * blockDim.x) {
    bool one;
    switch (mask_kind) {
      case 0: one = mask_is_one<int64_t>(mask, i); break;
      case 1: one = mask_is_one<float>(mask, i); break;
      case 2: one = mask_is_one<int32_t>(mask, i); break;
      case 3: one = reinterpret_cast<const uint16_t*>(mask)[i] == 0x3F80u; break;  // bf16 1.0
      case 4: one = reinterpret_cast<const uint16_t*>(mask)[i] == 0x3C00u; break;  // f16 1.0
      case 5: one = mask_is_one<uint8_t>(mask, i); break;
      default: one = mask_is_one<double>(mask, i); break;
    }
    bad |= !one;
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0 && bad_flag) {
    *bad_flag = 1;
    __threadfence_system();
  }
}

// ------------------------------------------------------------------ argmax over fp32 logits
__global__ void argmax_partial_kernel(unsigned long long* keys, const float* __restrict__ logits, long long V) {
  const int b = blockIdx.y;
  const float* row = logits + (size_t)b * V;
  unsigned long long best = 0ull;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < V;
       i += (long long)gridDim.x * blockDim.x) {
    unsigned long long k = argmax_key(row[i], (unsigned)i);
    best = k > best ? k : best;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  if ((threadIdx.x & 31) == 0 && best) atomicMax(&keys[b], best);
}
__global__ void argmax_final_kernel(int64_t* out, unsigned long long* keys, int B) {
  int b = threadIdx.x;
  if (b < B) { out[b] = (int64_t)argmax_key_index(keys[b]); keys[b] = 0ull; }
}

// ------------------------------------------------------------------ KV gather
template <typename T>
__global__ void kv_gather_kernel(T* __restrict__ out, const T* __restrict__ pool,
                                 const int32_t* __restrict__ page_table, int pt_stride, int page_size,
                                 int T_len, int nkv, int hd) {
  // out: [B, nkv, T, hd]; grid (T, B)
  const int j = blockIdx.x, b = blockIdx.y;
  const int page = page_table[(size_t)b * pt_stride + j / page_size];
  const T* src = pool + ((size_t)page * page_size + (j % page_size)) * (size_t)(nkv * hd);
  for (int u = threadIdx.x; u < nkv * hd; u += blockDim.x) {
    int kh = u / hd, d = u % hd;
    out[(((size_t)b * nkv + kh) * T_len + j) * hd + d] = src[u];
  }
}

}  // namespace pg

using namespace pg;

extern "C" {

const char* pg_last_error(void) { return g_err; }
int pg_abi_version(void) { return 1; }
unsigned long long pg_launch_count(void) { return g_launches.load(); }

int pg_set_next_prefetch(const void* ptr, long long bytes) {
  PG_REQUIRE(bytes >= 0 && ((uintptr_t)ptr % 16) == 0, "set_next_prefetch: region must be 16-byte aligned");
  g_prefetch = {(const char*)ptr, (unsigned long long)(ptr ? bytes : 0)};
  return PG_OK;
}

int pg_embed_merge(void* out, const int64_t* ids, const void* emb, const void* img_feats, int n_tokens,
                   int D, int64_t vocab, int64_t image_token_id, int64_t pad_id, int n_img_rows,
                   float img_div, float normalizer, int* err_flag, int dtype, void* stream) {
  return pg_embed_merge_ex(out, ids, emb, img_feats, n_tokens, D, vocab, image_token_id, pad_id, n_img_rows, img_div, normalizer,
                           err_flag, 0, nullptr, nullptr, dtype, stream);
}

int pg_embed_merge_ex(void* out, const int64_t* ids, const void* emb, const void* img_feats, int n_tokens,
                      int D, int64_t vocab, int64_t image_token_id, int64_t pad_id, int n_img_rows,
                      float img_div, float normalizer, int* err_flag, int drawn, const int32_t* step,
                      long long* info, int dtype, void* stream) {
  if (n_tokens <= 0) return PG_OK;
  PG_DISPATCH_DTYPE(dtype, T, {
    PG_REQUIRE(D % Vec<T>::N == 0, "embed_merge: D=%d not a multiple of %d", D, Vec<T>::N);
    embed_merge_kernel<T><<<n_tokens, 256, 0, (cudaStream_t)stream>>>(
        (T*)out, ids, (const T*)emb, (const T*)img_feats, n_tokens, D, vocab, image_token_id, pad_id,
        n_img_rows, img_div, normalizer, err_flag, drawn, step, info);
  });
  return check_launch("embed_merge");
}

int pg_rmsnorm(void* out, const void* x, const void* w, int rows, int D, float eps, int dtype, void* stream) {
  if (rows <= 0) return PG_OK;
  PG_DISPATCH_DTYPE(dtype, T, {
    constexpr int V = Vec<T>::N;
    PG_REQUIRE(D % V == 0 && D <= 256 * V * 4, "rmsnorm: unsupported D=%d", D);
    const T* none = nullptr;
    if (rows >= 64 && D <= 32 * V * 5)
      return launch_tc("rmsnorm", rows <= 1024 ? norm_rows_warp_kernel<T, 5, false, true> : norm_rows_warp_kernel<T, 5, false, false>,
                       dim3(cdiv(rows, rows <= 1024 ? 2 : 8)), dim3(rows <= 1024 ? 64 : 256), 0, 1, rows <= 4096,
                       (cudaStream_t)stream, (T*)out, (const T*)x, (const T*)w, none, rows, D, eps);
    if (rows >= 64 && D <= 32 * V * 8)
      return launch_tc("rmsnorm", rows <= 1024 ? norm_rows_warp_kernel<T, 8, false, true> : norm_rows_warp_kernel<T, 8, false, false>,
                       dim3(cdiv(rows, rows <= 1024 ? 2 : 8)), dim3(rows <= 1024 ? 64 : 256), 0, 1, rows <= 4096,
                       (cudaStream_t)stream, (T*)out, (const T*)x, (const T*)w, none, rows, D, eps);
    return launch_tc("rmsnorm", rmsnorm_kernel<T, 4>, dim3(rows), dim3(256), 0, 1, rows <= 1024, (cudaStream_t)stream, (T*)out,
                     (const T*)x, (const T*)w, D, eps);
  });
  return PG_OK;
}

int pg_layernorm(void* out, const void* x, const void* w, const void* b, int rows, int D, float eps,
                 int dtype, void* stream) {
  if (rows <= 0) return PG_OK;
  PG_DISPATCH_DTYPE(dtype, T, {
    constexpr int V = Vec<T>::N;
    PG_REQUIRE(D % V == 0 && D <= 256 * V * 4, "layernorm: unsupported D=%d", D);
    if (rows >= 64 && D <= 32 * V * 5)
      return launch_tc("layernorm", rows <= 1024 ? norm_rows_warp_kernel<T, 5, true, true> : norm_rows_warp_kernel<T, 5, true, false>,
                       dim3(cdiv(rows, rows <= 1024 ? 2 : 8)), dim3(rows <= 1024 ? 64 : 256), 0, 1, rows <= 4096,
                       (cudaStream_t)stream, (T*)out, (const T*)x, (const T*)w, (const T*)b, rows, D, eps);
    if (rows >= 64 && D <= 32 * V * 8)
      return launch_tc("layernorm", rows <= 1024 ? norm_rows_warp_kernel<T, 8, true, true> : norm_rows_warp_kernel<T, 8, true, false>,
                       dim3(cdiv(rows, rows <= 1024 ? 2 : 8)), dim3(rows <= 1024 ? 64 : 256), 0, 1, rows <= 4096,
                       (cudaStream_t)stream, (T*)out, (const T*)x, (const T*)w, (const T*)b, rows, D, eps);
    return launch_tc("layernorm", layernorm_kernel<T, 4>, dim3(rows), dim3(256), 0, 1, rows <= 1024, (cudaStream_t)stream,
                     (T*)out, (const T*)x, (const T*)w, (const T*)b, D, eps);
  });
  return PG_OK;
}

int pg_im2col(void* out, const void* pixels, int B, int C, int H, int W, int p, int ld_out, int dtype,
              void* stream) {
  PG_REQUIRE(H % p == 0 && W % p == 0 && ld_out >= C * p * p, "im2col: bad geometry");
  long long total = (long long)B * (H / p) * (W / p) * ld_out;
  if (total <= 0) return PG_OK;
  int grid = (int)((total + 255) / 256);
  if (grid > 148 * 16) grid = 148 * 16;
  const long long n_rows = (long long)B * (H / p) * (W / p) * C * p;
  PG_DISPATCH_DTYPE(dtype, T, {
    if (p % 2 == 0 && W % 2 == 0 && ld_out % 2 == 0 && ((uintptr_t)out | (uintptr_t)pixels) % (2 * sizeof(T)) == 0 && n_rows < (1ll << 31)) {
      im2col_rows_kernel<T><<<(int)(n_rows <= 148 * 64 * 256 ? (n_rows + 255) / 256 : 148 * 64), 256, 0, (cudaStream_t)stream>>>(
          (T*)out, (const T*)pixels, C, H, W, p, ld_out, (int)n_rows);
      return check_launch("im2col");
    }
    im2col_kernel<T><<<grid, 256, 0, (cudaStream_t)stream>>>((T*)out, (const T*)pixels, C, H, W, p, ld_out, total);
  });
  return check_launch("im2col");
}

int pg_rope_append(void* q_out, const void* qkv, const float* inv_freq, const int32_t* positions,
                   void* k_pool, void* v_pool, const int32_t* page_table, int pt_stride, int page_size,
                   const int32_t* slot_base, int B, int q_len, int nq, int nkv, int hd, int max_pos,
                   int dtype, void* stream) {
  if (B * q_len <= 0) return PG_OK;
  PG_REQUIRE(hd % 2 == 0, "rope_append: odd head_dim");
  PG_DISPATCH_DTYPE(dtype, T, {
    const uintptr_t any = (uintptr_t)q_out | (uintptr_t)qkv | (uintptr_t)k_pool | (uintptr_t)v_pool;
    if (hd % 4 == 0 && hd <= 1024 && any % (2 * sizeof(T)) == 0) {
      const int heads = nq + 2 * nkv, quarter = hd / 4;
      const int per = B * q_len <= 64 ? 1 : heads;               // heads per CTA
      const int groups = per == 1 ? 1 : min(min(4, heads), 256 / quarter);
      return launch_tc("rope_append", rope_append_pair_kernel<T>, dim3(B * q_len, cdiv(heads, per)), dim3(quarter * groups), 0, 1,
                       B * q_len <= 1024, (cudaStream_t)stream, (T*)q_out, (const T*)qkv, inv_freq, positions, (T*)k_pool,
                       (T*)v_pool, page_table, pt_stride, page_size, slot_base, q_len, nq, nkv, hd, max_pos, per);
    }
    return launch_tc("rope_append", rope_append_kernel<T>, dim3(B * q_len), dim3(256), 0, 1, B * q_len <= 1024,
                     (cudaStream_t)stream, (T*)q_out, (const T*)qkv, inv_freq, positions, (T*)k_pool, (T*)v_pool, page_table,
                     pt_stride, page_size, slot_base, q_len, nq, nkv, hd, max_pos);
  });
  return PG_OK;
}

int pg_step_advance(int64_t* next_ids, int64_t* history, int hist_stride, int* step_counter,
                    unsigned long long* keys, const int64_t* sampled, int32_t* kv_len, int32_t* positions,
                    int B, const pg_tp_exchange* keys_ex, void* stream) {
  PG_REQUIRE(B > 0 && B <= 1024, "step_advance: B=%d", B);
  const TpEx tex = tp_ex_from(keys_ex);
  PG_REQUIRE(!keys_ex || (tex.tp >= 2 && tex.tp <= TP_MAX_RANKS && (long long)B * 16 <= tex.slot_bytes),
             "step_advance: bad tensor-parallel key exchange");
  step_advance_kernel<<<1, ((B + 31) / 32) * 32, 0, (cudaStream_t)stream>>>(
      next_ids, history, hist_stride, step_counter, keys, sampled, kv_len, positions, B, tex);
  return check_launch("step_advance");
}

int pg_decode_inputs(int64_t* ids_dst, const int64_t* ids_src, int32_t* positions, int position, const void* mask,
                     int mask_kind, long long mask_n, int* bad_flag, int B, void* stream) {
  PG_REQUIRE(B > 0 && ids_dst && ids_src && positions, "decode_inputs: bad arguments");
  PG_REQUIRE(!mask || (mask_kind >= 0 && mask_kind <= 6), "decode_inputs: unknown mask element kind %d", mask_kind);
  // four mask elements per thread: one CTA walked the masks of 32 sequences of 389 tokens in 10.8 us
  const long long n = mask ? mask_n : 0;
  const int grid = n <= 1024 ? 1 : (n >= 148 * 1024 ? 148 : (int)((n + 1023) / 1024));
  decode_inputs_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(ids_dst, ids_src, positions, position, mask, mask_kind, n, bad_flag, B);
  return check_launch("decode_inputs");
}

int pg_argmax(int64_t* out, const float* logits, unsigned long long* keys, int B, int64_t V, void* stream) {
  PG_REQUIRE(B > 0 && B <= 1024, "argmax: B=%d", B);
  int gx = (int)((V + 256 * 8 - 1) / (256 * 8));
  if (gx > 148) gx = 148;
  argmax_partial_kernel<<<dim3(gx, B), 256, 0, (cudaStream_t)stream>>>(keys, logits, V);
  if (out) argmax_final_kernel<<<1, ((B + 31) / 32) * 32, 0, (cudaStream_t)stream>>>(out, keys, B);
  return check_launch("argmax");
}

int pg_kv_gather(void* out, const void* pool, const int32_t* page_table, int pt_stride, int page_size, int B,
                 int T_len, int nkv, int hd, int dtype, void* stream) {
  if (B * T_len <= 0) return PG_OK;
  PG_DISPATCH_DTYPE(dtype, T, {
    kv_gather_kernel<T><<<dim3(T_len, B), 128, 0, (cudaStream_t)stream>>>((T*)out, (const T*)pool, page_table,
                                                                          pt_stride, page_size, T_len, nkv, hd);
  });
  return check_launch("kv_gather");
}

}  // extern "C"
