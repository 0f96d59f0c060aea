// A decode step's narrow projections, up to 32 token rows, as an evenly shared weight stream: out[M, N] = X[M, K] W[N, K]^T + epilogue.
//
// What bounds them is the weight stream.  As tiles of 128 weight rows (gemm_tcgen05_skinny.cu) they are 16 to 20, whose K is cut over
// clusters that occupy 128 of the 148 SMs and meet through distributed shared memory; as rows of their own for one or two warps
// (gemv.cu) 512 CTAs do not come out even, and each warp's stream is short.  Here every SM takes the same number of weight rows, to
// within one: [N b / grid, N (b + 1) / grid), in groups of 16.  The 8 warps of a CTA split K, 128 columns of every 1024 each; weights
// go straight from global memory into mma.m16n8k16 B fragments with 16-byte loads (the contraction index is permuted alike for both
// operands: lane j of a quad owns 8 consecutive columns of every 32), about 128 KB of them in flight per SM, the first of them
// requested before the preceding launch has finished, as far as that leaves room: a CTA takes three quarters of an SM's registers,
// so between two streams a small launch (a norm) hides more than fusing it would save.  The tokens are the A operand, copied to shared memory: as a whole where a CTA
// has several groups, else each lane's own pieces, as many steps ahead as the weights (without that their trip to L2 bounds a step:
// K 16384, 8 rows 17.8 us, now 13.2).  Up to three rows take fp32 multiply-adds instead of mma.  The warps' partial sums meet in
// shared memory, in warp order.
#include "common.cuh"
#include "mma_frag.cuh"

namespace pg {

constexpr int GS_WARPS = 8, GS_KB = 4, GS_CHUNK = 32 * GS_KB * GS_WARPS;   // a chunk: GS_KB times 32 columns a warp
constexpr int GS_PAD = 32;                                                  // elements behind a row: a quarter-warp's rows meet no bank twice

struct StreamParams {
  void* C;
  const void* A;
  const void* W;
  const void* bias;
  const void* R;
  int M, N, K, lda, ldw, ldc, ldr, out_f32;
  int w_param;   // W is no output of a preceding launch: it may be requested before the dependency wait
};

template <typename T, int EPI>
__device__ __forceinline__ float stream_epilogue(const StreamParams& p, float s, int m, int n) {
  constexpr bool HAS_BIAS = EPI == PG_EPI_BIAS || EPI == PG_EPI_BIAS_GELU || EPI == PG_EPI_BIAS_RES;
  if (HAS_BIAS) s += to_f<T>(reinterpret_cast<const T*>(p.bias)[n]);
  float x = rnd<T>(s);
  if (EPI == PG_EPI_BIAS_GELU) x = rnd<T>(gelu_tanh_fast(x));
  if (EPI == PG_EPI_BIAS_RES || EPI == PG_EPI_RES) x = rnd<T>(x + to_f<T>(reinterpret_cast<const T*>(p.R)[(size_t)m * p.ldr + n]));
  return x;
}

constexpr int gs_ring(int mh, bool xs) { return !xs && mh == 4 ? 2 : 4; }

// MH: blocks of 8 token rows (1, 2 or 4).  NB: 0, or so many rows by fp32 multiply-adds instead of mma.  XS: all tokens' columns are in shared memory,
// otherwise those of RING items are, each lane's pieces copied by itself.
template <typename T, int EPI, int MH, bool XS, int NB>
__global__ void __launch_bounds__(GS_WARPS * 32, 1)
gemm_stream_kernel(StreamParams p) {
  constexpr int RING = gs_ring(MH, XS);               // items (a group's chunks, 2 GS_KB loads of a lane) in flight
  constexpr int MG = (MH + 1) / 2;                    // groups of 16 token rows
  constexpr int PART = GS_WARPS * MH * 8 * 16;
  extern __shared__ __align__(16) uint8_t smem[];     // part [2][warp][MH 8][16] fp32 | x: [M][K + pad], or [RING][warp][MH 8][128]
  float* part = reinterpret_cast<float*>(smem);
  T* xs = reinterpret_cast<T*>(smem + 2 * PART * sizeof(float));
  const int ldx = p.K + GS_PAD;
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, j = lane & 3;
  const int n0 = (int)((long long)p.N * blockIdx.x / gridDim.x), n1 = (int)((long long)p.N * (blockIdx.x + 1) / gridDim.x);
  const int chunks = (p.K + GS_CHUNK - 1) / GS_CHUNK, items = (n1 - n0 + 15) / 16 * chunks;
  const int col_w = warp * 32 * GS_KB + j * 8;        // this lane's first column in a chunk
  const T* W = reinterpret_cast<const T*>(p.W) + (size_t)(n0 + r) * p.ldw + col_w;
  const T* A = reinterpret_cast<const T*>(p.A) + (size_t)r * p.lda + col_w;
  const size_t second = (size_t)8 * p.ldw;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 ring[RING][2][GS_KB];
  int req = 0, req_chunk = 0, req_n = n0;             // the next item to request
  const T* req_row = W;
  auto request = [&](uint4 (&w)[2][GS_KB]) {
    const int col = req_chunk * GS_CHUNK;
    const bool live = req < items;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int b = 0; b < GS_KB; ++b) {
        const bool in = live && col_w + col + 32 * b < p.K && req_n + r + 8 * x < n1;
        w[x][b] = in ? ldg_stream(req_row + x * second + col + 32 * b) : zero;
      }
    ++req;
    if (++req_chunk == chunks) { req_chunk = 0; req_n += 16; req_row += (size_t)16 * p.ldw; }
  };
  if (!p.w_param) pdl_wait();
#pragma unroll
  for (int i = 0; i < RING; ++i) request(ring[i]);
  pdl_wait();                                         // the tokens, the residual and the output belong to the preceding kernels
  // without XS: piece b of a row in a slot; odd rows start 64 bytes on, so that a quarter-warp meets no bank twice
  auto slot = [&](int s, int row, int b) {
    return xs + ((size_t)(s * GS_WARPS + warp) * (MH * 8) + row) * (32 * GS_KB) + (((b * 4 + j) ^ ((row & 1) << 2)) * 8);
  };
  int copied = 0;                                     // the next item whose tokens are copied
  auto copy = [&](int s) {
    const int col = copied % chunks * GS_CHUNK;
#pragma unroll
    for (int h = 0; h < MH; ++h)
#pragma unroll
      for (int b = 0; b < GS_KB; ++b)
        if (copied < items && 8 * h + r < p.M && col_w + col + 32 * b < p.K)
          cp_async16(slot(s, 8 * h + r, b), A + (size_t)(8 * h) * p.lda + col + 32 * b);
    cp_async_commit();
    ++copied;
  };
  if (XS) {
    const int vecs = p.K / 8;
    for (int row = warp; row < p.M; row += GS_WARPS)
      for (int c = lane; c < vecs; c += 32) cp_async16(xs + (size_t)row * ldx + 8 * c, reinterpret_cast<const T*>(p.A) + (size_t)row * p.lda + 8 * c);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  } else {
#pragma unroll
    for (int i = 0; i < RING; ++i) copy(i);
  }

  float sum[NB > 0 ? NB : 1][2];                      // [token row][weight rows], with NB
#pragma unroll
  for (int t = 0; t < (NB > 0 ? NB : 1); ++t) sum[t][0] = sum[t][1] = 0.f;
  float acc[MG][2][2][4];                             // [token rows][weight rows][chain]
#pragma unroll
  for (int g = 0; g < MG; ++g)
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[g][x][0][e] = acc[g][x][1][e] = 0.f;
  int chunk = 0, buf = 0, n = n0;
  for (int i0 = 0; i0 < items; i0 += RING) {
#pragma unroll
    for (int d = 0; d < RING; ++d) {
      if (i0 + d >= items) break;                     // the same for the whole CTA
      if (!XS) cp_async_wait<RING - 1>();
      if constexpr (NB > 0) {
        static_assert(!XS && MH == 1, "rows of 8");
        __syncwarp();                                 // lanes of row t have copied it for all
#pragma unroll
        for (int b = 0; b < GS_KB; ++b) {
          float w[2][8];
          unpack<T>(ring[d][0][b], w[0]);
          unpack<T>(ring[d][1][b], w[1]);
          const bool in = chunk * GS_CHUNK + col_w + 32 * b < p.K;
#pragma unroll
          for (int t = 0; t < NB; ++t) {
            float x[8];
            unpack<T>(in ? *reinterpret_cast<const uint4*>(slot(d, t, b)) : zero, x);
#pragma unroll
            for (int e = 0; e < 8; ++e) { sum[t][0] = fmaf(w[0][e], x[e], sum[t][0]); sum[t][1] = fmaf(w[1][e], x[e], sum[t][1]); }
          }
        }
        __syncwarp();
      } else {
        uint4 xv[MH][GS_KB];
#pragma unroll
        for (int h = 0; h < MH; ++h)
#pragma unroll
          for (int b = 0; b < GS_KB; ++b) {
            const int col = chunk * GS_CHUNK + col_w + 32 * b;
            const T* at = XS ? xs + (size_t)(8 * h + r) * ldx + col : slot(d, 8 * h + r, b);
            xv[h][b] = 8 * h + r < p.M && col < p.K ? *reinterpret_cast<const uint4*>(at) : zero;
          }
#pragma unroll
        for (int b = 0; b < GS_KB; ++b)
#pragma unroll
          for (int g = 0; g < MG; ++g) {
            const uint4 a = xv[2 * g][b], c = 2 * g + 1 < MH ? xv[2 * g + 1 < MH ? 2 * g + 1 : 0][b] : zero;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const uint4& w = ring[d][x][b];
              mma_16816<T>(acc[g][x][0], a.x, c.x, a.y, c.y, w.x, w.y);
              mma_16816<T>(acc[g][x][1], a.z, c.z, a.w, c.w, w.z, w.w);
            }
          }
      }
      if (!XS) copy(d);
      request(ring[d]);
      if (++chunk < chunks) continue;
      // ---- the group's sums: acc[g][x][.][0..1] row 16 g + r, weight rows 8 x + 2 j and + 1; [2..3] row 16 g + r + 8
      float* mp = part + (size_t)buf * PART + (size_t)warp * (MH * 8 * 16);
      if constexpr (NB > 0) {
#pragma unroll
        for (int t = 0; t < NB; ++t)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            float v = sum[t][x];
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (j == 0) mp[t * 16 + x * 8 + r] = v;
            sum[t][x] = 0.f;
          }
      } else {
#pragma unroll
        for (int g = 0; g < MG; ++g)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            float* at = mp + (g * 16 + r) * 16 + x * 8 + 2 * j;
            auto& s = acc[g][x];
            *reinterpret_cast<float2*>(at) = make_float2(s[0][0] + s[1][0], s[0][1] + s[1][1]);
            if (2 * g + 1 < MH) *reinterpret_cast<float2*>(at + 8 * 16) = make_float2(s[0][2] + s[1][2], s[0][3] + s[1][3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) s[0][e] = s[1][e] = 0.f;
          }
      }
      __syncthreads();                                // the other buffer's readers are through as well
      for (int i = threadIdx.x; i < p.M * 16; i += GS_WARPS * 32) {
        const int m = i / 16, f = i % 16;
        if (n + f >= n1) continue;
        const float* at = part + (size_t)buf * PART + m * 16 + f;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < GS_WARPS; ++w) s += at[w * (MH * 8 * 16)];
        const float v = stream_epilogue<T, EPI>(p, s, m, n + f);
        if (p.out_f32) reinterpret_cast<float*>(p.C)[(size_t)m * p.ldc + n + f] = v;
        else reinterpret_cast<T*>(p.C)[(size_t)m * p.ldc + n + f] = from_f<T>(v);
      }
      buf ^= 1;
      chunk = 0;
      n += 16;
    }
  }
}

template <typename T, int EPI, int MH, bool XS, int NB = 0>
static int launch_stream(const StreamParams& p, int grid, cudaStream_t st) {
  const size_t x = XS ? (size_t)p.M * (p.K + GS_PAD) : (size_t)gs_ring(MH, XS) * MH * 8 * GS_CHUNK;
  const size_t smem = sizeof(float) * 2 * GS_WARPS * MH * 8 * 16 + sizeof(T) * x;
  return launch_pdl("gemm_stream", gemm_stream_kernel<T, EPI, MH, XS, NB>, dim3(grid), dim3(GS_WARPS * 32), smem, st, p);
}

static int stream_grid(int N) { return cdiv(N, 8) < 148 ? cdiv(N, 8) : 148; }

template <typename T, int EPI>
static int launch_stream_pick(const StreamParams& p, cudaStream_t st) {
  const int grid = stream_grid(p.N);
  if (cdiv(p.N, grid) > 16) return p.M <= 8 ? launch_stream<T, EPI, 1, true>(p, grid, st) : launch_stream<T, EPI, 2, true>(p, grid, st);
  if (p.M <= 8) return launch_stream<T, EPI, 1, false>(p, grid, st);
  if (p.M <= 16) return launch_stream<T, EPI, 2, false>(p, grid, st);
  return launch_stream<T, EPI, 4, false>(p, grid, st);
}

// One group a CTA (N up to 2368): up to 16 rows always, up to 32 where the two chunks of K 2048 hold their tokens (us, weights out of
// HBM, the tiles of 128 rows and this: 8 rows, N 2048 and K 16384 16.5 and 14.0, N 1024 and K 4096 5.6 and 4.2, N 128 and K 128 3.0 and
// 1.6; 16 rows of K 16384 16.6 and 15.9; 32 rows, N = K = 2048 4.9 and 4.8; 32 rows of K 16384 16.8 and 22).  Several groups, up to 4 (behind
// them the tiles' own stream is as even: gate/up of 16384 features 22.2 and 22.5), and up to 16 rows whose columns leave the loads in
// flight their L1: from K 512 on (8 rows, N 8192: K 512 4.8 and 4.9, but K 448 3.8 and 4.9, where the warps of a CTA whose columns lie
// behind K only wait), up to K 3072 for 8 rows and K 5120 for more, whose second block of tokens the tiles pay for as well; at 4 groups 1024
// less (8 rows, N 2560: K 2048 5.5 and 4.6, 3584 6.8 and 8.0; N 8192: K 2048 9.7 and 9.8, 2560 10.9 and 12.6).  The upper lines were drawn
// when the tiles handed their sums round in four times the time; they are ahead of this a little below them now (8 rows, N 2560,
// K 3072 6.1 and 6.4; 12 rows, N 2560: K 3072 6.1 and 6.6, 5120 8.8 and 9.1; 16 rows, N 8192, K 512 4.9 and 5.6), which the rule does not
// use yet.
bool gemm_stream_wanted(int M, int N, int K, int epi) {
  if (M < 4 || M > 32 || epi < PG_EPI_NONE || epi > PG_EPI_RES) return false;
  const int groups = cdiv(cdiv(N, stream_grid(N)), 16);
  if (groups == 1) return M <= 16 || K <= 2 * GS_CHUNK;
  if (groups > 4 || M > 16 || K < 512 || K > (M <= 8 ? 3072 : 5120) - (groups == 4 ? 1024 : 0)) return false;
  return 2 * (size_t)M * (K + GS_PAD) <= 136 * 1024;
}

// One to three rows of a decode step (o_proj and down_proj): rows of x, out and R lie K, N and N apart; R may be NULL.
template <typename T>
static int gemv_stream_t(const StreamParams& p, int grid, cudaStream_t st) {
  if (p.R) {
    if (p.M == 1) return launch_stream<T, PG_EPI_RES, 1, false, 1>(p, grid, st);
    if (p.M == 2) return launch_stream<T, PG_EPI_RES, 1, false, 2>(p, grid, st);
    return launch_stream<T, PG_EPI_RES, 1, false, 3>(p, grid, st);
  }
  if (p.M == 1) return launch_stream<T, PG_EPI_NONE, 1, false, 1>(p, grid, st);
  if (p.M == 2) return launch_stream<T, PG_EPI_NONE, 1, false, 2>(p, grid, st);
  return launch_stream<T, PG_EPI_NONE, 1, false, 3>(p, grid, st);
}

// Against one warp a row, from K 8192 on two (gemv_res_kernel), weights out of HBM, us there and here.  A short row leaves the warps of
// a CTA without columns (N = 2048: one row of K 512 2.0 and 2.6, of K 2048 3.5 and 3.3, 4096 6.2 and 4.8; with up to 64 CTAs earlier:
// N 512, K 768 2.0 and 1.7; three rows, whose products bound a warp, from K 1024: 3.4 and 3.1).  From K 8192 on two and three rows of
// few features come out faster there (three rows of K 16384: N 1024 14.4 and 15.7, N 2048, more CTAs than find room at once, 28.0
// and 17.4; two rows: N 256 10.5 and 11.4, N 768 12.6 and 11.7; one row of N 2048 14.2 and 12.3).
bool gemv_stream_wanted(int B, int N, int K) {
  if (B < 1 || B > 3 || K % 8 || cdiv(N, stream_grid(N)) > 16) return false;
  if (K >= 8192) return B == 1 || N >= (B == 2 ? 768 : 148 * 3 * 4);
  return K >= 2048 || (B == 3 && K >= 1024) || (N <= 512 && K >= 640);
}

int gemv_stream(void* out, const void* x, const void* W, const void* R, int B, int N, int K, int dtype, cudaStream_t st) {
  const StreamParams p = {out, x, W, nullptr, R, B, N, K, K, K, N, N, 0, 1};
  return dtype == PG_BF16 ? gemv_stream_t<bf16>(p, stream_grid(N), st) : gemv_stream_t<f16>(p, stream_grid(N), st);
}

// 16-bit operands, N, K and leading dimensions multiples of 8, 16-byte aligned rows (checked by the caller)
int gemm_stream(void* C, const void* A, const void* W, const void* bias, const void* R, int M, int N, int K, int lda, int ldw, int ldc,
                int ldr, int epi, int out_f32, int dtype, bool w_param, cudaStream_t st) {
  const StreamParams p = {C, A, W, bias, R, M, N, K, lda, ldw, ldc, ldr, out_f32, w_param ? 1 : 0};
#define PG_ST(E) return dtype == PG_BF16 ? launch_stream_pick<bf16, E>(p, st) : launch_stream_pick<f16, E>(p, st)
  switch (epi) {
    case PG_EPI_NONE: PG_ST(PG_EPI_NONE);
    case PG_EPI_BIAS: PG_ST(PG_EPI_BIAS);
    case PG_EPI_BIAS_GELU: PG_ST(PG_EPI_BIAS_GELU);
    case PG_EPI_BIAS_RES: PG_ST(PG_EPI_BIAS_RES);
    case PG_EPI_RES: PG_ST(PG_EPI_RES);
  }
#undef PG_ST
  set_error("gemm_stream: bad epilogue %d", epi);
  return PG_ERR_INVALID;
}

}  // namespace pg
