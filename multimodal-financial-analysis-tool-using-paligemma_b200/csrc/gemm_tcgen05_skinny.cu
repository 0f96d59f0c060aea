// Skinny GEMM for batched decode (4 <= M <= 128 token rows): out[M,N] = X[M,K] W[N,K]^T.
// With so few rows the problem is a weight stream, so the operands are swapped: the WEIGHT tile is the 128-row
// A operand of tcgen05.mma and the tokens are the N dimension (N_mma = M rounded up to 16).  A pipeline stage is
// then 16 KB of weights + a few KB of activations, so 8-10 stages (~150 KB of weights) are in flight per SM —
// what a 6 TB/s stream needs — instead of the 16 KB-activation/8 KB-weight stages of the row-major kernel.
// The accumulator is D^T: TMEM lane = output feature, column = token.
//   S == 1 : persistent over the N/128 weight tiles (gate/up with the GeGLU pairing, lm_head), double-buffered
//            accumulators so the epilogue overlaps the next tile's stream; a thread keeps its feature, so bias is one scalar
//            and the stores are coalesced across the warp (consecutive features of one token);
//   S  > 1 : a cluster of S CTAs splits K for one weight tile (q/k/v, o_proj, down_proj have 16-20 tiles only).  Every CTA
//            leaves its partial tile in its shared memory, a row per token, and finishes the S-th part of the tokens from all
//            of them, four neighbouring features a lane (distributed shared memory, summed in rank order).  With S = 8 a CTA
//            keeps to half an SM's shared memory: clusters of 8 whole SMs do not all fit the GPCs at once.
// o_proj and down_proj (K 2048 and 16384) together, weights out of HBM: the pair kernel with a workspace and a reduce launch each
// (gemm_tcgen05_swap.cu) 25.4 us for 8 rows and 26.3 for 32, this 21.6 and 22.0.
#include "tc_common.cuh"

namespace pg {
namespace tc {

constexpr int SN_BM = 128, SN_BK = 64;

struct SnParams {
  void* C;
  const void* bias;
  const void* R;
  int M, N, K, ldc, ldr, out_f32;
  int w_param;   // W is no output of a preceding launch: it may be requested before the dependency wait
};

template <bool DUAL, int NT, int S>
constexpr int sn_stages() {
  constexpr int bytes = (DUAL ? 2 : 1) * SN_BM * SN_BK * 2 + (NT * SN_BK * 2 + 1023) / 1024 * 1024;
  constexpr int n = (S == 8 ? 100 : 200) * 1024 / bytes;
  return n > 10 ? 10 : n;
}

// NT: token columns of the accumulator (multiple of 16, <= 256).  S: K split (cluster size).
template <typename T, int EPI, int NT, int S>
__global__ void __launch_bounds__(256, S == 8 ? 2 : 1)
gemm_tc_skinny_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, SnParams p) {
  constexpr bool DUAL = (EPI == PG_EPI_GEGLU);
  constexpr int NW = DUAL ? 2 : 1;                               // weight tiles per stage
  constexpr int W_BYTES = SN_BM * SN_BK * 2, X_BYTES = NT * SN_BK * 2;
  constexpr int X_PAD = (X_BYTES + 1023) / 1024 * 1024;          // keep every tile 1024-byte aligned
  constexpr int STAGE_BYTES = NW * W_BYTES + X_PAD;
  constexpr int NSTAGES = sn_stages<DUAL, NT, S>();
  constexpr int ACC_COLS = NW * NT;                              // TMEM columns per accumulator stage
  constexpr int TMEM_COLS = 2 * ACC_COLS <= 32 ? 32 : (2 * ACC_COLS <= 64 ? 64 : (2 * ACC_COLS <= 128 ? 128 : (2 * ACC_COLS <= 256 ? 256 : 512)));
  static_assert(2 * ACC_COLS <= 512, "accumulators do not fit TMEM");
  constexpr uint32_t IDESC = umma_idesc(std::is_same<T, bf16>::value ? 1 : 0, SN_BM, NT);

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = smem_base + NSTAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (NSTAGES + s); };
  auto tfull_bar = [&](int a) { return bars + 8u * (2 * NSTAGES + a); };
  auto tempty_bar = [&](int a) { return bars + 8u * (2 * NSTAGES + 2 + a); };
  const uint32_t tmem_slot = bars + 8u * (2 * NSTAGES + 4);
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  // S > 1: fp32 partial D, one padded row per token ([NT][128 + 4]), reusing the ring
  constexpr int PROW = SN_BM + 4;
  static_assert(S == 1 || NT * PROW * 4 <= NSTAGES * STAGE_BYTES, "the partial tile does not fit the stage ring");
  float* part = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = S > 1 ? cluster_rank() : 0;
  const int n_tiles = (p.N + SN_BM - 1) / SN_BM;
  const int k_blocks = (p.K + SN_BK - 1) / SN_BK, per = (k_blocks + S - 1) / S;
  const int kb0 = (int)crank * per, kb1 = min(k_blocks, kb0 + per);
  const int tile_first = (S > 1) ? (int)(blockIdx.x / S) : (int)blockIdx.x;
  const int tile_stride = (S > 1) ? n_tiles : (int)gridDim.x;      // S > 1: exactly one tile per cluster

  if (warp == 1 && lane == 0) {
    for (int s = 0; s < NSTAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), 4); }
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
    // ===================== TMA producer: weight tile(s) + the token block =====================
    // flat item index i -> (tile, k block).  The first NSTAGES items' WEIGHT tiles are requested before
    // griddepcontrol.wait: a parameter does not depend on the preceding kernel, so ~150 KB per SM is already in flight
    // when the predecessor's activations become visible; the token blocks follow the wait.
    if (!p.w_param) pdl_wait();
    const int nk = kb1 - kb0;
    const int my_tiles = tile_first < n_tiles ? (n_tiles - tile_first + tile_stride - 1) / tile_stride : 0;
    const int items = my_tiles * nk;
    auto item_tile = [&](int i) { return tile_first + (i / nk) * tile_stride; };
    auto item_kb = [&](int i) { return kb0 + i % nk; };
    const int pre = items < NSTAGES ? items : NSTAGES;
    for (int i = 0; i < pre; ++i) {                               // fresh barriers: every stage is free
      const uint32_t sa = smem_base + i * STAGE_BYTES;
      mbar_expect_tx(full_bar(i), NW * W_BYTES + X_BYTES);
      tma_load_2d(sa, &map_w, full_bar(i), item_kb(i) * SN_BK, item_tile(i) * SN_BM);
      if (DUAL) tma_load_2d(sa + W_BYTES, &map_w, full_bar(i), item_kb(i) * SN_BK, p.N + item_tile(i) * SN_BM);
    }
    pdl_wait();
    for (int i = 0; i < pre; ++i)
      tma_load_2d(smem_base + i * STAGE_BYTES + NW * W_BYTES, &map_x, full_bar(i), item_kb(i) * SN_BK, 0);
    int stage = pre == NSTAGES ? 0 : pre;
    uint32_t phase = pre == NSTAGES ? 1 : 0;
    for (int i = pre; i < items; ++i) {
      mbar_wait(empty_bar(stage), phase ^ 1);
      const uint32_t sa = smem_base + stage * STAGE_BYTES;
      mbar_expect_tx(full_bar(stage), NW * W_BYTES + X_BYTES);
      tma_load_2d(sa, &map_w, full_bar(stage), item_kb(i) * SN_BK, item_tile(i) * SN_BM);
      if (DUAL) tma_load_2d(sa + W_BYTES, &map_w, full_bar(stage), item_kb(i) * SN_BK, p.N + item_tile(i) * SN_BM);
      tma_load_2d(sa + NW * W_BYTES, &map_x, full_bar(stage), item_kb(i) * SN_BK, 0);
      if (++stage == NSTAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1 && lane == 0) {
    // ===================== MMA issuer: D^T[128 features, NT tokens] += W_tile X_tile^T =====================
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    for (int tile = tile_first; tile < n_tiles; tile += tile_stride) {
      mbar_wait(tempty_bar(acc), acc_phase ^ 1);
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(full_bar(stage), phase);
        tc_fence_after();
        const uint32_t sa = smem_base + stage * STAGE_BYTES;
#pragma unroll
        for (int k = 0; k < SN_BK / 16; ++k) {
          const uint64_t xd = umma_desc(sa + NW * W_BYTES + k * 32);
          const uint32_t accumulate = (kb > kb0 || k > 0) ? 1u : 0u;
          umma(d_tmem, umma_desc(sa + k * 32), xd, IDESC, accumulate);
          if (DUAL) umma(d_tmem + NT, umma_desc(sa + W_BYTES + k * 32), xd, IDESC, accumulate);
        }
        umma_commit(empty_bar(stage));
        if (++stage == NSTAGES) { stage = 0; phase ^= 1; }
      }
      umma_commit(tfull_bar(acc));
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }
  __syncwarp();

  // ===================== epilogue: thread <-> output feature, columns <-> tokens =====================
  const int q = warp & 3, r = q * 32 + lane;
  const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
  T* Ct = reinterpret_cast<T*>(p.C);
  float* Cf = reinterpret_cast<float*>(p.C);
  const T* bias = reinterpret_cast<const T*>(p.bias);
  const T* R = reinterpret_cast<const T*>(p.R);
  if (warp >= 4) pdl_wait();   // residual reads / output writes only after the predecessor has finished
  auto finish = [&](int tile, float (&v)[16], float (&u)[DUAL ? 16 : 1], int m0) {
    const int n = tile * SN_BM + r;
    if (n >= p.N) return;
    float bn = 0.f;
    if (EPI == PG_EPI_BIAS || EPI == PG_EPI_BIAS_GELU || EPI == PG_EPI_BIAS_RES) bn = to_f<T>(bias[n]);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int m = m0 + j;
      if (m >= p.M) break;
      float x = rnd<T>(v[j] + bn);
      if (EPI == PG_EPI_BIAS_GELU) x = rnd<T>(gelu_tanh_fast(x));
      if (EPI == PG_EPI_GEGLU) x = rnd<T>(rnd<T>(gelu_tanh_fast(x)) * rnd<T>(u[DUAL ? j : 0]));
      if (EPI == PG_EPI_BIAS_RES || EPI == PG_EPI_RES) x = rnd<T>(x + to_f<T>(R[(size_t)m * p.ldr + n]));
      if (p.out_f32) Cf[(size_t)m * p.ldc + n] = x;
      else Ct[(size_t)m * p.ldc + n] = from_f<T>(x);
    }
  };

  if constexpr (S == 1) {
    if (warp >= 4) {
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int tile = tile_first; tile < n_tiles; tile += tile_stride) {
        mbar_wait(tfull_bar(acc), acc_phase);
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < NT / 16; ++c) {
          float v[16], u[DUAL ? 16 : 1];
          tmem_ld16(t_lane + acc * ACC_COLS + c * 16, v);
          if (DUAL) tmem_ld16(t_lane + acc * ACC_COLS + NT + c * 16, u);
          tmem_ld_wait();
          finish(tile, v, u, c * 16);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(acc));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    const int tile = tile_first;
    const bool have_k = kb1 > kb0;
    // This CTA finishes NC of the tokens: a warp one of them at a time, four neighbouring features a lane.  (A feature's row per lane
    // made every load of a warp 32 lines of the peer's shared memory: 32 rows, N 2048, K 16384 by 8 19.6 us, now 16.8; N 2560, K 2048
    // 8.7, now 5.6.)  All NC tokens go round, whether the matrix has them or not: 17 rows cost what 32 do.
    constexpr int NC = NT / S, STEPS = NC / 4;
    const int m0 = (int)crank * NC + (warp & 3), f = 4 * lane, n = tile * SN_BM + f;
    constexpr bool HAS_BIAS = EPI == PG_EPI_BIAS || EPI == PG_EPI_BIAS_GELU || EPI == PG_EPI_BIAS_RES;
    constexpr bool HAS_RES = EPI == PG_EPI_BIAS_RES || EPI == PG_EPI_RES;
    float res[STEPS][4], bn[4] = {0.f, 0.f, 0.f, 0.f};
    auto four = [&](const T* at, float (&v)[4]) {
      const uint2 u = __ldg(reinterpret_cast<const uint2*>(at));   // gemm_tc takes rows on 16-byte boundaries only
      unpack_pair<T>(u.x, v);
      unpack_pair<T>(u.y, v + 2);
    };
    if (warp >= 4) {
      // bias and residual are requested before the accumulator is waited for (N is a multiple of 8)
      if (HAS_BIAS && n < p.N) four(bias + n, bn);
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        res[i][0] = res[i][1] = res[i][2] = res[i][3] = 0.f;
        if (HAS_RES && n < p.N && m0 + 4 * i < p.M) four(R + (size_t)(m0 + 4 * i) * p.ldr + n, res[i]);
      }
      mbar_wait(tfull_bar(0), 0);   // this CTA's MMAs are complete: accumulator final, stage ring idle
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < NT / 16; ++c) {
        float v[16];
        tmem_ld16(t_lane + c * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) part[(c * 16 + j) * PROW + r] = have_k ? v[j] : 0.f;
      }
    }
    tc_fence_before();
    cluster_sync_all();
    float v[STEPS][4];
    if (warp >= 4) {
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        float4 pv[S];
#pragma unroll
        for (int peer = 0; peer < S; ++peer) {        // all loads in flight before the first add
          const int at = (m0 + 4 * i) * PROW + f;
          pv[peer] = peer == (int)crank ? *reinterpret_cast<const float4*>(part + at) : ld_dsmem_v4(smem_base + (uint32_t)(at * 4), peer);
        }
        v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.f;
#pragma unroll
        for (int peer = 0; peer < S; ++peer) { v[i][0] += pv[peer].x; v[i][1] += pv[peer].y; v[i][2] += pv[peer].z; v[i][3] += pv[peer].w; }
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // this warp has read its peers' shared memory
    if (warp >= 4 && n < p.N) {
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        const int m = m0 + 4 * i;
        if (m >= p.M) break;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x = rnd<T>(v[i][j] + bn[j]);
          if (EPI == PG_EPI_BIAS_GELU) x = rnd<T>(gelu_tanh_fast(x));
          if (HAS_RES) x = rnd<T>(x + res[i][j]);
          v[i][j] = x;
        }
        if (p.out_f32) {
          *reinterpret_cast<float4*>(Cf + (size_t)m * p.ldc + n) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
        } else {
          *reinterpret_cast<uint2*>(Ct + (size_t)m * p.ldc + n) = make_uint2(pack_pair<T>(v[i][0], v[i][1]), pack_pair<T>(v[i][2], v[i][3]));
        }
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");     // nobody leaves while a peer may still read its shared memory
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

template <typename T, int EPI, int NT, int S>
static int launch_sn(const CUtensorMap& mx, const CUtensorMap& mw, const SnParams& p, cudaStream_t st) {
  constexpr bool DUAL = (EPI == PG_EPI_GEGLU);
  constexpr int X_PAD = (NT * SN_BK * 2 + 1023) / 1024 * 1024;
  constexpr int STAGE_BYTES = (DUAL ? 2 : 1) * SN_BM * SN_BK * 2 + X_PAD;
  constexpr int NSTAGES = sn_stages<DUAL, NT, S>();
  const size_t smem = 1024 + (size_t)NSTAGES * STAGE_BYTES + 8 * (2 * NSTAGES + 4) + 16;
  auto kern = gemm_tc_skinny_kernel<T, EPI, NT, S>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    set_error("gemm_tc_skinny: cannot reserve %zu B of shared memory", smem);
    cudaGetLastError();
    return PG_ERR_CUDA;
  }
  const int n_tiles = cdiv(p.N, SN_BM);
  const int grid = S > 1 ? n_tiles * S : (n_tiles < 148 ? n_tiles : 148);
  return launch_tc("gemm_tcgen05_skinny", kern, dim3(grid), dim3(256), smem, S, true, st, mx, mw, p);
}

template <typename T, int EPI, int NT>
static int launch_sn_s(const CUtensorMap& mx, const CUtensorMap& mw, const SnParams& p, int s, cudaStream_t st) {
  if (EPI != PG_EPI_GEGLU) {
    if (s == 8) return launch_sn<T, (EPI == PG_EPI_GEGLU ? PG_EPI_NONE : EPI), NT, 8>(mx, mw, p, st);
    if (s == 4) return launch_sn<T, (EPI == PG_EPI_GEGLU ? PG_EPI_NONE : EPI), NT, 4>(mx, mw, p, st);
    if (s == 2) return launch_sn<T, (EPI == PG_EPI_GEGLU ? PG_EPI_NONE : EPI), NT, 2>(mx, mw, p, st);
  }
  return launch_sn<T, EPI, NT, 1>(mx, mw, p, st);
}

template <typename T, int EPI>
static int launch_sn_nt(const CUtensorMap& mx, const CUtensorMap& mw, const SnParams& p, int nt, int s, cudaStream_t st) {
  if (nt <= 32) return launch_sn_s<T, EPI, 32>(mx, mw, p, s, st);
  if (nt <= 64) return launch_sn_s<T, EPI, 64>(mx, mw, p, s, st);
  return launch_sn_s<T, EPI, 128>(mx, mw, p, s, st);
}

}  // namespace tc

bool gemm_tc_skinny_wanted(int M, int N, int K, int epi) {
  // Weights out of HBM, this and the split row-major kernel, us.  Up to 32 rows the swap-AB stream takes every projection that
  // gemm_stream.cu leaves (32 rows: gate/up 28.0 and 31.1, lm_head 172 and 184, N 2560, K 2048 5.6 and 7.0).  Up to 64 rows it does
  // so for long K (64 rows, N 2048, K 8192 12.1 and 15.5).  The line at K was drawn when the merge of 64 columns cost four times
  // what it does now (N 2560, K 2048 13.8 and 11.9 then); today this kernel would be ahead below it too (6.9 and 7.7; N 1152, K 4304
  // 8.3 and 9.6, the pair kernel that takes it 9.0; N = K = 2048 with a residual 6.4 and 7.2, the pair kernel 8.0), which the rule does not use
  // yet.  Above, only where CTAs own whole weight tiles or there are 32 of them (128 rows: N = K = 4096 12.6 and 13.3; N 2560, K 2048
  // 11.4 and 9.2).
  static const int mode = env_int("PG_SKINNY", 1);   // 0 off, 1 where it wins, 2 everywhere it applies
  if (!mode || M < 4 || M > 128 || N < 512 || K < 256 || epi < PG_EPI_NONE || epi > PG_EPI_GEGLU) return false;
  if (mode == 2) return true;
  const int n_tiles = cdiv(N, 128);
  if (epi == PG_EPI_GEGLU || n_tiles >= 100 || M <= 32) return true;
  return M <= 64 ? K >= (epi == PG_EPI_NONE ? 4096 : 8192) : epi == PG_EPI_NONE && n_tiles >= 32 && K >= 4096;
}

// Split of K across a cluster until ~148 CTAs stream (each keeps >= 4 K blocks).  A CTA of a cluster of 4 takes an SM's whole shared
// memory, and no more than 32 such clusters find room at once (N 4304, K 1152, 8 rows: 34 clusters 8.7 us, pairs 5.2)
int gemm_tc_skinny_split(int N, int K, int epi) {
  const int n_tiles = cdiv(N, tc::SN_BM), kb = cdiv(K, tc::SN_BK);
  int s = 1;
  if (epi != PG_EPI_GEGLU)
    while (s < 8 && n_tiles * s * 2 <= (s == 2 ? 128 : 160) && kb / (s * 2) >= 4) s *= 2;
  return s;
}

int gemm_tc_skinny(void* C, const void* A, const void* W, const void* bias, const void* R, int M, int N, int K, int lda,
                   int ldw, int ldc, int ldr, int epi, int out_f32, int dtype, bool w_param, cudaStream_t st) {
  const bool bf = dtype == PG_BF16;
  const int nt = M <= 32 ? 32 : (M <= 64 ? 64 : 128), s = gemm_tc_skinny_split(N, K, epi);
  CUtensorMap mx, mw;
  const int w_rows = (epi == PG_EPI_GEGLU) ? 2 * N : N;
  PG_REQUIRE(tc::make_map_2d(&mx, A, M, K, lda, nt, bf) && tc::make_map_2d(&mw, W, w_rows, K, ldw, tc::SN_BM, bf),
             "gemm_tc_skinny: cuTensorMapEncodeTiled failed");
  tc::SnParams p = {C, bias, R, M, N, K, ldc, ldr, out_f32, w_param};
#define PG_SN(E) return bf ? tc::launch_sn_nt<bf16, E>(mx, mw, p, nt, s, st) : tc::launch_sn_nt<f16, E>(mx, mw, p, nt, s, st)
  switch (epi) {
    case PG_EPI_NONE: PG_SN(PG_EPI_NONE);
    case PG_EPI_BIAS: PG_SN(PG_EPI_BIAS);
    case PG_EPI_BIAS_GELU: PG_SN(PG_EPI_BIAS_GELU);
    case PG_EPI_BIAS_RES: PG_SN(PG_EPI_BIAS_RES);
    case PG_EPI_RES: PG_SN(PG_EPI_RES);
    case PG_EPI_GEGLU: PG_SN(PG_EPI_GEGLU);
  }
#undef PG_SN
  set_error("gemm_tc_skinny: bad epilogue %d", epi);
  return PG_ERR_INVALID;
}

}  // namespace pg
