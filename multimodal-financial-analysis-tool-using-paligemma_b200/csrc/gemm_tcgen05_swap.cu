// Prompt-sized GEMMs (129..512 token rows: the 260-token prefill and the cache-off recompute of the KV ablation):
// C[M,N] = A[M,K] W[N,K]^T with the operands SWAPPED on CTA pairs.
//
// With a few hundred token rows every nn.Linear of the Gemma decoder is a weight-streaming problem (5 GB of weights
// against 1e12 FLOP), but the row-major kernels treat the tokens as the 128-row MMA operand: 260 rows make three
// m-tiles (the third 97 % padding), the weights are re-read per m-tile out of L2 and the L2 -> SM fabric (~6300 B/clk
// chip-wide), not HBM or the tensor pipe, sets the time (gate/up 48 us, down_proj 56 us per layer).  Here:
//   * the WEIGHT rows are the M = 256 operand of a tcgen05.mma.cta_group::2 (128 rows per CTA of the pair), streamed
//     from HBM exactly once;
//   * ALL tokens are the N operand: one accumulator of NT <= 256 columns (<= 256 tokens) or a second one for the rest (<= 512 tokens) at
//     TMEM column 256; the pair SPLITS the token tile (each CTA stages NT/2 token rows per k-block), so the token re-read that
//     every weight tile costs is halved against single-CTA swap-AB;
//   * short-N / long-K problems (o_proj, down_proj, q/k/v: 8-10 weight tiles) are split along K over the 74 pairs;
//     every work item leaves an fp32 partial [split][token][feature] in a caller-provided workspace (L2-resident) and
//     gemm_swap_reduce_kernel sums the splits and applies the epilogue (residual / GeGLU / rounding points of
//     gemm_simt.cu) with fully coalesced rows.
// Roles per CTA (as gemm_tcgen05_2cta.cu): warp 0 TMA producer, warp 1 (leader CTA) MMA issuer, warp 2 TMEM
// allocation, warps 4-11 epilogue (TMEM -> 16 tokens x 128 features in shared memory -> fp32 partial sums by TMA store).
// The four staging buffers take 32 KB of the ring: 5 stages of 33 KB at 260 rows, 3 of 47 to 48 KB from 481 rows on (6 and 4 without).
// With them, down_proj (N 2048, K 16384), us: 129 rows 25.0 -> 20.3, 260 33.0 -> 26.4, 384 38.0 -> 31.0, 448 41.0 -> 33.7,
// 512 44.4 -> 38.9; N 640 at 512 rows 28.9 -> 20.5.
#include "tc_common.cuh"

namespace pg {
namespace tc {

constexpr int SW_BK = 64, SW_WROWS = 128, SW_THREADS = 384;
constexpr int SW_W_BYTES = SW_WROWS * SW_BK * 2;   // 16 KB of weights per CTA per k-block
constexpr int SW_OUT_BYTES = 16 * SW_WROWS * 4;    // 16 tokens' partial sums of a CTA's 128 features
constexpr int SW_SMEM_BUDGET = 220 * 1024 - 4 * SW_OUT_BYTES;

struct ParamsSw {
  float* P;            // workspace: [splits][M tokens][N features] fp32
  int M, N, K;         // tokens, output features, reduction length
  int NT, NT2;         // widths of the first and the second token tile (multiples of 16, <= 256; NT2 may be 0)
  int splits, kb_per_split, stages;
  int w_param;         // W is no output of a preceding launch: it may be requested before the dependency wait
};

__device__ __forceinline__ uint32_t sw_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void sw_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void sw_tma_cg2(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void sw_umma_cg2(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void sw_commit_cg2(uint32_t bar, uint16_t cta_mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(cta_mask) : "memory");
}

template <int FMT>  // 1 bf16, 0 f16
__global__ void __launch_bounds__(SW_THREADS, 1)
gemm_swap_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                 const __grid_constant__ CUtensorMap map_x2, const __grid_constant__ CUtensorMap map_p, ParamsSw p) {
  constexpr int MAX_STAGES = 8;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int x_bytes = (p.NT / 2) * SW_BK * 2;                 // the first token tile's half per k-block (multiple of 1024)
  const int stage_bytes = SW_W_BYTES + ((p.NT + p.NT2) / 2) * SW_BK * 2;
  const uint32_t out_base = smem_base + p.stages * stage_bytes, bars = out_base + 4 * SW_OUT_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };                      // used in the leader CTA
  auto empty_bar = [&](int s) { return bars + 8u * (MAX_STAGES + s); };      // one per CTA
  const uint32_t tfull_bar = bars + 8u * (2 * MAX_STAGES);                   // one per CTA
  const uint32_t tempty_bar = bars + 8u * (2 * MAX_STAGES + 1);              // used in the leader CTA
  const uint32_t tmem_slot = bars + 8u * (2 * MAX_STAGES + 2);
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t crank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  const bool leader = crank == 0;
  const int f_tiles = (p.N + 2 * SW_WROWS - 1) / (2 * SW_WROWS);
  const int items = f_tiles * p.splits;
  const int first = (int)(blockIdx.x / 2), stride = (int)(gridDim.x / 2);
  const int k_blocks = (p.K + SW_BK - 1) / SW_BK;
  const uint32_t idesc = umma_idesc(FMT, 2 * SW_WROWS, p.NT), idesc2 = umma_idesc(FMT, 2 * SW_WROWS, p.NT2 ? p.NT2 : 16);

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_x)) : "memory");
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(tfull_bar, 1);
    mbar_init(tempty_bar, 16);  // 8 epilogue warps x 2 CTAs
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers and TMEM exist before anything lands on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  if (warp == 0) {
    // ===================== TMA producer (both CTAs): own 128 weight rows + own half of every token tile =====================
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool waited = false;
      if (!p.w_param) { pdl_wait(); waited = true; }
      for (int item = first; item < items; item += stride) {
        const int ft = item / p.splits, sp = item % p.splits;
        const int kb0 = sp * p.kb_per_split, kb1 = min(k_blocks, kb0 + p.kb_per_split);
        // every pair walks its k-blocks from a different starting point: at any moment the pairs read different
        // token slices, so the few hundred L2 lines of one slice are not requested by all 148 SMs at once
        const int nkb = kb1 - kb0, rot = (first * 5) % nkb;
        for (int i = 0; i < nkb; ++i) {
          const int kb = kb0 + (i + rot) % nkb;
          mbar_wait(empty_bar(stage), phase ^ 1);
          const uint32_t sa = smem_base + stage * stage_bytes;
          const uint32_t full_leader = sw_mapa(full_bar(stage), 0);
          if (leader) mbar_expect_tx(full_bar(stage), 2 * stage_bytes);  // both CTAs' bytes
          // a parameter does not depend on the preceding kernels: its first load goes out before the dependency wait
          sw_tma_cg2(sa, &map_w, full_leader, kb * SW_BK, ft * 2 * SW_WROWS + (int)crank * SW_WROWS);
          if (!waited) { pdl_wait(); waited = true; }   // the token rows come from the predecessor
          sw_tma_cg2(sa + SW_W_BYTES, &map_x, full_leader, kb * SW_BK, (int)crank * (p.NT / 2));
          if (p.NT2) sw_tma_cg2(sa + SW_W_BYTES + x_bytes, &map_x2, full_leader, kb * SW_BK, p.NT + (int)crank * (p.NT2 / 2));
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
      }
      if (!waited) pdl_wait();
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (leader CTA only) =====================
    if (leader && lane == 0) {
      int stage = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int item = first; item < items; item += stride) {
        const int sp = item % p.splits;
        const int kb0 = sp * p.kb_per_split, kb1 = min(k_blocks, kb0 + p.kb_per_split);
        mbar_wait(tempty_bar, acc_phase ^ 1);  // both CTAs' epilogues have drained the accumulator
        tc_fence_after();
        for (int i = kb0; i < kb1; ++i) {      // the producer's k order (rotated per pair); the sum does not care
          mbar_wait(full_bar(stage), phase);
          tc_fence_after();
          const uint32_t sa = smem_base + stage * stage_bytes;
#pragma unroll
          for (int k = 0; k < SW_BK / 16; ++k) {
            const uint32_t accumulate = (i > kb0 || k > 0) ? 1u : 0u;
            sw_umma_cg2(tmem_base, umma_desc(sa + k * 32), umma_desc(sa + SW_W_BYTES + k * 32), idesc, accumulate);
            if (p.NT2) sw_umma_cg2(tmem_base + 256, umma_desc(sa + k * 32), umma_desc(sa + SW_W_BYTES + x_bytes + k * 32), idesc2, accumulate);
          }
          sw_commit_cg2(empty_bar(stage), (uint16_t)0x3);  // the stage is free in BOTH CTAs once these MMAs have read it
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        sw_commit_cg2(tfull_bar, (uint16_t)0x3);           // accumulator complete, in both CTAs' TMEM
        acc_phase ^= 1;
      }
    }
  } else if (warp >= 4) {
    // ===================== epilogue: TMEM -> fp32 partial [split][token][feature] (both CTAs) =====================
    // A chunk of 16 tokens goes to shared memory as 16 rows of 128 features and on by one TMA store of the warpgroup's first thread;
    // two buffers for each of the two warpgroups.  (A feature per lane and a store per token: 6.7 us of the 28 of 260 rows, N 2048, K 16384; a
    // 260-token prompt with its image, with the reduction below asking for all splits at once, 3985 -> 3920 us.)
    const int q = warp & 3, half = (warp - 4) >> 2;  // TMEM lane quarter; the two halves interleave 16-column chunks
    const bool store_thread = q == 0 && lane == 0;
    uint32_t acc_phase = 0;
    const int chunks_per_tile = p.NT / 16, chunks = chunks_per_tile + p.NT2 / 16;
    uint8_t* const out_sm = smem_raw + (out_base - smem_u32(smem_raw)) + half * 2 * SW_OUT_BYTES;
    pdl_wait();  // the workspace may still be read by the predecessor's reduce kernel
    int buf = 0;
    for (int item = first; item < items; item += stride) {
      const int ft = item / p.splits, sp = item % p.splits;
      const int f0 = ft * 2 * SW_WROWS + (int)crank * SW_WROWS;   // this CTA's first output feature
      mbar_wait(tfull_bar, acc_phase);
      tc_fence_after();
      const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
      for (int c = half; c < chunks; c += 2, buf ^= 1) {
        const int t = c >= chunks_per_tile ? 1 : 0, cc = c - t * chunks_per_tile;   // the second token tile lives from TMEM column 256 on
        float v[16];
        tmem_ld16(t_lane + t * 256 + cc * 16, v);
        if (store_thread) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // the buffer's last store has read it
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        tmem_ld_wait();
        float* row = reinterpret_cast<float*>(out_sm + buf * SW_OUT_BYTES) + q * 32 + lane;
#pragma unroll
        for (int j = 0; j < 16; ++j) row[j * SW_WROWS] = v[j];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        if (store_thread) {
          if (f0 < p.N)
            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"   // clipped at N and at M
                         ::"l"(reinterpret_cast<uint64_t>(&map_p)), "r"(out_base + (half * 2 + buf) * SW_OUT_BYTES), "r"(f0),
                         "r"(t * p.NT + cc * 16), "r"(sp) : "memory");
          // A group for every chunk, be it empty: the wait above counts groups.  Without one for the chunks of a CTA whose features
          // lie past N, the group it lets pend is the last store of the item before, out of the buffer that is written next.
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) sw_arrive_cluster(sw_mapa(tempty_bar, 0));
      acc_phase ^= 1;
    }
    if (store_thread) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the leader's MMAs read this CTA's shared memory, its commits arrive on this CTA's barriers
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

// out[m][n] = epilogue(sum over splits of P[s][m][n]); rounding points of gemm_simt.cu / gemm_tc_kernel.
// GeGLU: W = [Wgate; Wup], P has 2*Nout columns, out[m][f] = rnd(rnd(gelu(rnd(g))) * rnd(u)).
template <typename T, int EPI>
__global__ void __launch_bounds__(256)
gemm_swap_reduce_kernel(T* __restrict__ out, const float* __restrict__ P, const T* __restrict__ R, int M, int Nout, int Np,
                        int splits, int ldc, int ldr) {
  pdl_launch_dependents();
  pdl_wait();
  const int vec_per_row = Nout / 4;
  const long long total = (long long)M * vec_per_row;
  const size_t split_stride = (size_t)M * Np;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int m = (int)(i / vec_per_row), n = (int)(i % vec_per_row) * 4;
    const float* src = P + (size_t)m * Np + n;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), u = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int AT_ONCE = EPI == PG_EPI_GEGLU ? 4 : 10;      // splits whose loads are in flight together
    for (int s0 = 0; s0 < splits; s0 += AT_ONCE) {
      float4 v[AT_ONCE], w[EPI == PG_EPI_GEGLU ? AT_ONCE : 1];
#pragma unroll
      for (int k = 0; k < AT_ONCE; ++k)
        if (s0 + k < splits) {
          v[k] = __ldcg(reinterpret_cast<const float4*>(src + (s0 + k) * split_stride));
          if (EPI == PG_EPI_GEGLU) w[EPI == PG_EPI_GEGLU ? k : 0] = __ldcg(reinterpret_cast<const float4*>(src + (s0 + k) * split_stride + Nout));
        }
#pragma unroll
      for (int k = 0; k < AT_ONCE; ++k)
        if (s0 + k < splits) {
          a.x += v[k].x; a.y += v[k].y; a.z += v[k].z; a.w += v[k].w;
          if (EPI == PG_EPI_GEGLU) {
            const float4 x = w[EPI == PG_EPI_GEGLU ? k : 0];
            u.x += x.x; u.y += x.y; u.z += x.z; u.w += x.w;
          }
        }
    }
    float o[4] = {rnd<T>(a.x), rnd<T>(a.y), rnd<T>(a.z), rnd<T>(a.w)};
    if (EPI == PG_EPI_GEGLU) {
      const float uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = rnd<T>(rnd<T>(gelu_tanh_fast(o[j])) * rnd<T>(uu[j]));
    }
    if (EPI == PG_EPI_RES) {
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = rnd<T>(o[j] + to_f<T>(R[(size_t)m * ldr + n + j]));
    }
    T* dst = out + (size_t)m * ldc + n;
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[j] = from_f<T>(o[j]);
  }
}

}  // namespace tc

// ---------------------------------------------------------------------------------------- host side
static void* g_ws_ptr = nullptr;
static long long g_ws_bytes = 0;
static thread_local bool g_force_swap = false;   // pg_gemm(impl = 3): take this kernel for every epilogue it supports

void gemm_tc_swap_force(bool on) { g_force_swap = on; }

extern "C" int pg_set_workspace(void* ptr, long long bytes) {
  g_ws_ptr = ptr;
  g_ws_bytes = ptr ? bytes : 0;
  return PG_OK;
}

static void swap_plan(int M, int N, int K, tc::ParamsSw* p) {
  p->M = M; p->N = N; p->K = K;
  p->NT = M >= 256 ? 256 : (M + 15) / 16 * 16;
  p->NT2 = (M - (M < 256 ? M : 256) + 15) / 16 * 16;
  const int f_tiles = cdiv(N, 2 * tc::SW_WROWS), k_blocks = cdiv(K, tc::SW_BK);
  // split K until the work items fill the 74 CTA pairs about once (every split keeps >= 2 k-blocks)
  int splits = 1;
  if (f_tiles < 74) {
    splits = 74 / f_tiles;
    if (splits > k_blocks / 2) splits = k_blocks / 2 > 0 ? k_blocks / 2 : 1;
  }
  int kbs = cdiv(k_blocks, splits);
  splits = cdiv(k_blocks, kbs);           // no empty split
  p->splits = splits;
  p->kb_per_split = kbs;
  const int stage_bytes = tc::SW_W_BYTES + ((p->NT + p->NT2) / 2) * tc::SW_BK * 2;
  int stages = (tc::SW_SMEM_BUDGET - 1024 - 256) / stage_bytes;
  p->stages = stages > 8 ? 8 : stages;
  static const int max_stages = env_int("PG_SWAP_STAGES", 8);
  if (p->stages > max_stages) p->stages = max_stages;
}

// the partial sums [splits][M][N] fp32, for stores of 16 tokens x 128 features
static bool make_map_partials(CUtensorMap* map, void* base, int N, int M, int splits) {
  tc::EncodeTiledFn fn = tc::encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)splits};
  cuuint64_t strides[2] = {(cuuint64_t)N * 4, (cuuint64_t)M * N * 4};
  cuuint32_t box[3] = {tc::SW_WROWS, 16, 1}, estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool gemm_tc_swap_wanted(int M, int N, int K, int epi, int out_f32, int res_mod) {
  static const int enabled = env_int("PG_GEMM_SWAP", 1);
  static const int min_m = env_int("PG_GEMM_SWAP_MIN_M", 4);
  if ((!enabled && !g_force_swap) || out_f32 || res_mod != 0 || M < min_m || M > 512) return false;
  if (epi != PG_EPI_NONE && epi != PG_EPI_RES && epi != PG_EPI_GEGLU) return false;
  // which projections take this kernel (measured per projection): bit 0 q/k/v (no epilogue),
  // bit 1 o_proj (residual, K < 8192), bit 2 down_proj (residual, K >= 8192), bit 3 gate/up (GeGLU)
  // measured, us, weights out of HBM: prompt-sized rows (129..512) -- down_proj only (260 rows: 26.2, split over clusters 46.4; but
  // q/k/v 12.9 and 9.8, o_proj 12.3 and 10.0, gate/up 54 and 38 on the row-major kernels); batched-decode rows (33..128) -- o_proj
  // and down_proj (128 rows: o_proj 8.7 and 8.8, N 1152, K 4304 9.3 and 10.9, down_proj 20.3 and 28.3; at 64 rows o_proj 8.0, split by 4
  // 7.2 since its exchange is faster, which the rule does not use yet).  Up to 32 rows, and up to 64 with a long K, the cluster split
  // of gemm_tcgen05_skinny.cu is faster: it needs no workspace round trip (32 rows: 5.0 and 7.4, K 16384 16.8 and 18.9)
  static const int mask_large = env_int("PG_SWAP_MASK", 4), mask_small = env_int("PG_SWAP_MASK_SMALL", 6);
  if ((M <= 32 || (M <= 64 && K >= 8192)) && !g_force_swap) return false;
  const int mask = M > 128 ? mask_large : mask_small;
  const int kind = epi == PG_EPI_NONE ? 1 : (epi == PG_EPI_GEGLU ? 8 : (K >= 8192 ? 4 : 2));
  if (!(mask & kind) && !g_force_swap) return false;
  const int n_w = epi == PG_EPI_GEGLU ? 2 * N : N;   // weight rows
  if (n_w % 4 || N % 4) return false;
  tc::ParamsSw p;
  swap_plan(M, n_w, K, &p);
  if (p.stages < 3) return false;
  return g_ws_ptr && (uintptr_t)g_ws_ptr % 16 == 0 && (long long)p.splits * M * n_w * 4 <= g_ws_bytes;
}

int gemm_tc_swap(void* C, const void* A, const void* W, const void* R, int M, int N, int K, int lda, int ldw, int ldc,
                 int ldr, int epi, int dtype, bool w_param, cudaStream_t st) {
  const bool bf = dtype == PG_BF16;
  const int n_w = epi == PG_EPI_GEGLU ? 2 * N : N;
  tc::ParamsSw p;
  swap_plan(M, n_w, K, &p);
  p.P = reinterpret_cast<float*>(g_ws_ptr);
  p.w_param = w_param;
  CUtensorMap mw, mx, mx2 = {}, mp;
  PG_REQUIRE(tc::make_map_2d(&mw, W, n_w, K, ldw, tc::SW_WROWS, bf) && tc::make_map_2d(&mx, A, M, K, lda, p.NT / 2, bf) &&
                 (!p.NT2 || tc::make_map_2d(&mx2, A, M, K, lda, p.NT2 / 2, bf)) &&
                 make_map_partials(&mp, p.P, n_w, M, p.splits),
             "gemm_swap: cuTensorMapEncodeTiled failed (M=%d N=%d K=%d lda=%d ldw=%d)", M, n_w, K, lda, ldw);
  const int stage_bytes = tc::SW_W_BYTES + ((p.NT + p.NT2) / 2) * tc::SW_BK * 2;
  const size_t smem = 1024 + (size_t)p.stages * stage_bytes + 4 * tc::SW_OUT_BYTES + 8 * (2 * 8 + 3) + 16;
  auto kern = bf ? tc::gemm_swap_kernel<1> : tc::gemm_swap_kernel<0>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    set_error("gemm_swap: cannot reserve %zu B of shared memory", smem);
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  const int items = cdiv(n_w, 2 * tc::SW_WROWS) * p.splits;
  int rc = launch_tc("gemm_tcgen05_swap", kern, dim3(2 * (items < 74 ? items : 74)), dim3(tc::SW_THREADS), smem, 2, true, st,
                     mw, mx, mx2, mp, p);
  if (rc != PG_OK) return rc;
  const long long vecs = (long long)M * (N / 4);
  const int grid = (int)((vecs + 255) / 256 < 148 * 8 ? (vecs + 255) / 256 : 148 * 8);
#define PG_SWR(T_, E_)                                                                                          \
  return launch_tc("gemm_swap_reduce", tc::gemm_swap_reduce_kernel<T_, E_>, dim3(grid), dim3(256), 0, 1, true, st, \
                   (T_*)C, (const float*)p.P, (const T_*)R, M, N, n_w, p.splits, ldc, ldr)
  if (bf) {
    if (epi == PG_EPI_NONE) { PG_SWR(bf16, PG_EPI_NONE); }
    if (epi == PG_EPI_RES) { PG_SWR(bf16, PG_EPI_RES); }
    PG_SWR(bf16, PG_EPI_GEGLU);
  } else {
    if (epi == PG_EPI_NONE) { PG_SWR(f16, PG_EPI_NONE); }
    if (epi == PG_EPI_RES) { PG_SWR(f16, PG_EPI_RES); }
    PG_SWR(f16, PG_EPI_GEGLU);
  }
#undef PG_SWR
}

}  // namespace pg
