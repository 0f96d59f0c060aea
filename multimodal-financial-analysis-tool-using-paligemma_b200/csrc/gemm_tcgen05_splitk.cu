// Split-K companion of gemm_tcgen05.cu for GEMMs with few output tiles (prefill with a few hundred tokens: o_proj, q/k/v;
// SigLIP at batch 1; batched decode).  With 128-row tiles a 260 x 2048 output has 48-96 tiles, so part of the 148 SMs idles
// while the others pull all the operands through their own L2 port (about 64 B a clock, which is what paces these shapes).
// Here a cluster of S CTAs shares one output tile: CTA r runs the TMA -> tcgen05.mma pipeline over its 1/S of K into its own
// TMEM accumulator, leaves its fp32 partial tile in its shared memory, and after one cluster barrier every CTA finishes the
// S-th part of the tile's columns from all partials (distributed shared memory, summed in rank order) with the fused epilogue.
// A CTA keeps to less than half an SM's shared memory, so that the clusters of a whole wave find room in any GPC.
// No atomics, no global workspace, deterministic summation order.
#include "tc_common.cuh"

namespace pg {
namespace tc {

constexpr int SK_BM = 128, SK_BK = 64, SK_STAGES = 4;

struct SkParams {
  void* C;
  const void* bias;
  const void* R;
  int M, N, K, ldc, ldr, res_mod, out_f32;
  int w_param;   // W is no output of a preceding launch: it may be requested before the dependency wait
};

template <typename T, int EPI, int BN, int S>
__global__ void __launch_bounds__(256, 2)
gemm_tc_splitk_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, SkParams p) {
  constexpr int A_BYTES = SK_BM * SK_BK * 2, W_BYTES = BN * SK_BK * 2, STAGE_BYTES = A_BYTES + W_BYTES;
  constexpr int TMEM_COLS = BN < 32 ? 32 : BN;
  constexpr uint32_t IDESC = umma_idesc(std::is_same<T, bf16>::value ? 1 : 0, SK_BM, BN);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = smem_base + SK_STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (SK_STAGES + s); };
  const uint32_t tfull_bar = bars + 8u * (2 * SK_STAGES), tmem_slot = tfull_bar + 8;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  constexpr int PROW = BN + 4;   // [128][PROW] fp32 (16-byte accesses of neighbouring rows meet no bank twice), reuses the stage ring
  static_assert(128 * PROW * 4 <= SK_STAGES * STAGE_BYTES, "the partial tile does not fit the stage ring");
  float* part = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int tile = blockIdx.x / S;
  const int m_tiles = (p.M + SK_BM - 1) / SK_BM;
  const int n_blk = tile / m_tiles, m_blk = tile % m_tiles;
  const int k_blocks = (p.K + SK_BK - 1) / SK_BK, per = (k_blocks + S - 1) / S;
  const int kb0 = (int)rank * per, kb1 = min(k_blocks, kb0 + per);

  if (warp == 1 && lane == 0) {
    for (int s = 0; s < SK_STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(tfull_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  if (warp == 0 && lane == 0) {
    // a parameter does not depend on the preceding kernels: the ring's first weight tiles go out before the dependency wait
    if (!p.w_param) pdl_wait();
    const int pre = min(SK_STAGES, max(0, kb1 - kb0));
    for (int i = 0; i < pre; ++i) {
      mbar_expect_tx(full_bar(i), STAGE_BYTES);
      tma_load_2d(smem_base + i * STAGE_BYTES + A_BYTES, &map_w, full_bar(i), (kb0 + i) * SK_BK, n_blk * BN);
    }
    pdl_wait();
    for (int i = 0; i < pre; ++i) tma_load_2d(smem_base + i * STAGE_BYTES, &map_a, full_bar(i), (kb0 + i) * SK_BK, m_blk * SK_BM);
    int stage = pre == SK_STAGES ? 0 : pre;
    uint32_t phase = pre == SK_STAGES ? 1 : 0;
    for (int kb = kb0 + pre; kb < kb1; ++kb) {
      mbar_wait(empty_bar(stage), phase ^ 1);
      const uint32_t sa = smem_base + stage * STAGE_BYTES;
      mbar_expect_tx(full_bar(stage), STAGE_BYTES);
      tma_load_2d(sa, &map_a, full_bar(stage), kb * SK_BK, m_blk * SK_BM);
      tma_load_2d(sa + A_BYTES, &map_w, full_bar(stage), kb * SK_BK, n_blk * BN);
      if (++stage == SK_STAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1 && lane == 0) {
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(full_bar(stage), phase);
      tc_fence_after();
      const uint32_t sa = smem_base + stage * STAGE_BYTES;
#pragma unroll
      for (int k = 0; k < SK_BK / 16; ++k)
        umma(tmem_base, umma_desc(sa + k * 32), umma_desc(sa + A_BYTES + k * 32), IDESC, (kb > kb0 || k > 0) ? 1u : 0u);
      umma_commit(empty_bar(stage));
      if (++stage == SK_STAGES) { stage = 0; phase ^= 1; }
    }
    umma_commit(tfull_bar);
  }
  __syncwarp();
  // Out of TMEM two threads own a row (half of its columns each); the finished part goes by 16 bytes of a row to neighbouring lanes.
  const int q = warp & 3, r = q * 32 + lane, hf = warp >> 2;
  const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
  const bool have_k = kb1 > kb0;
  constexpr int NC = BN / S, HB = BN / 2;                   // columns that this CTA finishes; a half
  constexpr int LANES = NC / 4, ROWS = 32 / LANES, STEPS = 16 / ROWS;   // per row; rows of a warp at once; the warps' steps through 128 rows
  static_assert(HB == 32 && NC % 8 == 0 && STEPS >= 1, "a half is one load of TMEM");
  const int col = 4 * (lane % LANES), row0 = warp * ROWS + lane / LANES, m0 = m_blk * SK_BM + row0, n = n_blk * BN + (int)rank * NC + col;
  constexpr bool HAS_BIAS = EPI == PG_EPI_BIAS || EPI == PG_EPI_BIAS_GELU || EPI == PG_EPI_BIAS_RES;
  constexpr bool HAS_RES = EPI == PG_EPI_BIAS_RES || EPI == PG_EPI_RES;
  uint2 res[STEPS], bia = make_uint2(0, 0);
  pdl_wait();                 // residual reads / output writes only after the predecessor has finished
  if (HAS_BIAS && n < p.N) bia = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const T*>(p.bias) + n));   // N is a multiple of 8
#pragma unroll
  for (int i = 0; i < STEPS; ++i) {     // requested before the accumulator is waited for
    const int m = m0 + i * (8 * ROWS), rm = p.res_mod > 0 ? (m % p.res_mod) : m;
    res[i] = HAS_RES && m < p.M && n < p.N ? __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const T*>(p.R) + (size_t)rm * p.ldr + n))
                                           : make_uint2(0, 0);
  }
  mbar_wait(tfull_bar, 0);    // every MMA of this CTA has completed: accumulator final, stage ring idle
  __syncwarp();
  tc_fence_after();
  {
    float v[HB];
    tmem_ld32(t_row + hf * HB, v);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < HB; j += 4)
      *reinterpret_cast<float4*>(&part[r * PROW + hf * HB + j]) =
          have_k ? make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  tc_fence_before();
  cluster_sync_all();         // partial tiles are visible cluster-wide, and nobody reads TMEM any more
  // Whole row pieces by neighbouring lanes: with a row per lane each load of a warp is 32 lines of the peer's shared memory, and the
  // exchange took 3.1 us of the 8.4 between a launch's dependency and its end (256 rows, N 4304, K 1152 by 2).  The cluster is told that the
  // reads are done before the epilogue's arithmetic.  One image's 9 layers 544 -> 470 us, a 260-token prompt with its image
  // 4285 -> 3985.
  float4 pv[STEPS][S];
  auto read = [&](int i) {
    const int at = (row0 + i * (8 * ROWS)) * PROW + (int)rank * NC + col;
#pragma unroll
    for (int peer = 0; peer < S; ++peer)
      pv[i][peer] = peer == (int)rank ? *reinterpret_cast<const float4*>(part + at) : ld_dsmem_v4(smem_base + (uint32_t)(at * 4), peer);
  };
  if ((m_blk + 1) * SK_BM <= p.M) {
#pragma unroll
    for (int i = 0; i < STEPS; ++i) read(i);
  } else {                    // rows that nobody asked for cost the exchange as much as others
#pragma unroll
    for (int i = 0; i < STEPS; ++i) {
#pragma unroll
      for (int peer = 0; peer < S; ++peer) pv[i][peer] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m0 + i * (8 * ROWS) < p.M) read(i);
    }
  }
  float o[STEPS][4];
#pragma unroll
  for (int i = 0; i < STEPS; ++i) {
    o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
#pragma unroll
    for (int peer = 0; peer < S; ++peer) { o[i][0] += pv[i][peer].x; o[i][1] += pv[i][peer].y; o[i][2] += pv[i][peer].z; o[i][3] += pv[i][peer].w; }
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // this warp has read its peers' shared memory
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
  T* Ct = reinterpret_cast<T*>(p.C);
  float* Cf = reinterpret_cast<float*>(p.C);
  float bb[4];
  unpack_pair<T>(bia.x, bb);
  unpack_pair<T>(bia.y, bb + 2);
#pragma unroll
  for (int i = 0; i < STEPS; ++i) {
    const int m = m0 + i * (8 * ROWS);
    if (m >= p.M || n >= p.N) break;
    float rr[4];
    unpack_pair<T>(res[i].x, rr);
    unpack_pair<T>(res[i].y, rr + 2);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x = o[i][j];
      if (HAS_BIAS) x += bb[j];
      x = rnd<T>(x);
      if (EPI == PG_EPI_BIAS_GELU) x = rnd<T>(gelu_tanh_fast(x));
      if (HAS_RES) x = rnd<T>(x + rr[j]);
      o[i][j] = x;
    }
    if (p.out_f32) *reinterpret_cast<float4*>(Cf + (size_t)m * p.ldc + n) = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
    else *reinterpret_cast<uint2*>(Ct + (size_t)m * p.ldc + n) = make_uint2(pack_pair<T>(o[i][0], o[i][1]), pack_pair<T>(o[i][2], o[i][3]));
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // nobody leaves while a peer may still read its shared memory
}

template <typename T, int EPI, int BN, int S>
static int launch_sk(const CUtensorMap& ma, const CUtensorMap& mw, const SkParams& p, cudaStream_t st) {
  const size_t smem = 1024 + (size_t)SK_STAGES * (SK_BM * SK_BK * 2 + BN * SK_BK * 2) + 8 * (2 * SK_STAGES + 2) + 16;
  auto kern = gemm_tc_splitk_kernel<T, EPI, BN, S>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    set_error("gemm_tc_splitk: cannot reserve %zu B of shared memory", smem);
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  const int tiles = cdiv(p.M, SK_BM) * cdiv(p.N, BN);
  return launch_tc("gemm_tcgen05_splitk", kern, dim3(tiles * S), dim3(256), smem, S, true, st, ma, mw, p);
}

template <typename T, int EPI>
static int launch_sk_pick(const CUtensorMap& ma, const CUtensorMap& mw, const SkParams& p, int s, cudaStream_t st) {
  return s == 4 ? launch_sk<T, EPI, 64, 4>(ma, mw, p, st) : launch_sk<T, EPI, 64, 2>(ma, mw, p, st);
}

}  // namespace tc

// Split factor for a problem (0 = do not split): up to three m-tiles whose 64-wide tiles leave room for the split within one
// wave of two CTAs per SM, and at least 8 K blocks per CTA.  256 rows, weights out of HBM, whole and split, us: N 3456, K 1152
// 8.2 and 7.8; N = K = 2048 13.3 and 10.0; N 1152, K 4304 23.3 and 12.9.  By 4 with fewer than 16 K blocks a CTA only while three
// quarters of a wave are left free: the second CTA of an SM then gave away what the halved chain gains (256 rows, N = K = 2048: by 4
// 12.6, by 2 11.4 us, when a row of a peer's tile was read by one lane; by whole row pieces 9.7 and 10.0, within what two runs
// differ, so the line stands).  The limit of three m-tiles is from that time too: beyond it (385 rows: N = K = 2048 13.4 us whole,
// N 1152, K 4304 23.3) no split has been measured.  Gated pairings stay out: two accumulators a tile already fill the wave.
int gemm_tc_splitk_factor(int M, int N, int K, int epi) {
  static const int mode = env_int("PG_SPLITK", -1);   // 0 never, 2 / 4: that factor wherever it fits
  if (mode == 0 || epi == PG_EPI_GEGLU || epi == PG_EPI_SWIGLU || M > 3 * tc::SK_BM) return 0;
  const int kb = cdiv(K, tc::SK_BK), tiles = cdiv(M, tc::SK_BM) * cdiv(N, 64);
  for (int s = mode > 1 ? mode : 4; s >= 2; s /= 2)
    if (kb / s >= 8 && tiles * s <= (s >= 4 && kb / s < 16 ? 192 : 288)) return s;
  return 0;
}

int gemm_tc_splitk(void* C, const void* A, const void* W, const void* bias, const void* R, int M, int N, int K, int lda,
                   int ldw, int ldc, int ldr, int res_mod, int epi, int out_f32, int dtype, int s, bool w_param, cudaStream_t st) {
  const bool bf = dtype == PG_BF16;
  CUtensorMap ma, mw;
  PG_REQUIRE(tc::make_map_2d(&ma, A, M, K, lda, tc::SK_BM, bf) && tc::make_map_2d(&mw, W, N, K, ldw, 64, bf),
             "gemm_tc_splitk: cuTensorMapEncodeTiled failed");
  tc::SkParams p = {C, bias, R, M, N, K, ldc, ldr, res_mod, out_f32, w_param};
#define PG_SK(E) return bf ? tc::launch_sk_pick<bf16, E>(ma, mw, p, s, st) : tc::launch_sk_pick<f16, E>(ma, mw, p, s, st)
  switch (epi) {
    case PG_EPI_NONE: PG_SK(PG_EPI_NONE);
    case PG_EPI_BIAS: PG_SK(PG_EPI_BIAS);
    case PG_EPI_BIAS_GELU: PG_SK(PG_EPI_BIAS_GELU);
    case PG_EPI_BIAS_RES: PG_SK(PG_EPI_BIAS_RES);
    case PG_EPI_RES: PG_SK(PG_EPI_RES);
  }
#undef PG_SK
  set_error("gemm_tc_splitk: bad epilogue %d", epi);
  return PG_ERR_INVALID;
}

}  // namespace pg
