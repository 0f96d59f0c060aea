// Grouped expert GEMM for a decode step's few rows (up to 64 routed rows in all): out[pos] = A[pos] W_e^T for the rows of every
// expert that has some, with the pairings and roundings of moe_gemm_tcgen05.cu.
//
// With so few rows the product is a stream of the met experts' weights, and what bounds it is how evenly the SMs share that
// stream: tiles of 128 weight rows are 16 an expert, 160 for ten experts, two rounds on 148 SMs, and each also carries 128 rows of
// activations of which one or two count.  Here a unit is 16 weight rows (16 output features, or the gate and up rows of 8), so that
// a CTA of the persistent grid has 9 to 18 of them and the last round costs little.  The 8 warps of a CTA split K: each takes 128
// columns of every 1024, straight from global memory into mma.m16n8k16 B fragments with 16-byte loads (the contraction index is
// permuted alike for both operands: lane j of a quad owns 8 consecutive columns of every 32), 128 KB of them in flight per SM; the
// rows of A are in shared memory and are the A operand, up to 16 of one expert at a time (an expert with more has its weights read
// again).  The warps' partial sums meet in shared memory, in warp order.
// 16 rows, 10 of 16 experts met, K 2048: gate/up of 2048 features 57 -> 36 us, down 35 -> 19 (5.1 TB/s); 2 rows 29 and 16 -> 9 and 6.
// Measured against it: rows of A through L1 instead (no limit on them, but each unit waits for its loads: 39 and 28 us), 16 warps
// with half the columns each (33 and 23 us where this takes 30 and 19), units of 8 rows for down (20).
#include "common.cuh"
#include "mma_frag.cuh"

namespace pg {

constexpr int MF_PAIRS = 64, MF_ROWS = 16, MF_WARPS = 8, MF_KB = 4;
constexpr int MF_CHUNK = 32 * MF_KB * MF_WARPS;      // columns of a chunk: MF_KB times 32 a warp
constexpr int MF_RING = 4;                           // items (a unit's chunks, 2 MF_KB loads of a lane) in flight
constexpr int MF_PAD = 32;                           // elements behind a row: a quarter-warp's rows meet no bank twice
constexpr int MF_PART = MF_WARPS * MF_ROWS * 16;     // floats of a unit's partial sums

struct MoeFewParams {
  void* out;
  const void* A;
  const void* W;
  const int32_t* offsets;
  int ldo, lda, n_pairs, n_experts, N, K, act;
  float limit;
};

// One output value from its sum(s): the rounding points of moe_gemm_simt_kernel.
template <typename T, bool DUAL>
__device__ __forceinline__ float moe_few_activate(const MoeFewParams& p, float x, float u) {
  if (!DUAL && p.act == PG_ACT_RELU2) { x = fmaxf(x, 0.f); return x * x; }
  x = rnd<T>(x);
  if (DUAL) {
    float uu = rnd<T>(u);
    if (p.act == PG_GLU_CLAMPED) {
      x = fminf(x, p.limit);
      uu = fminf(fmaxf(uu, -p.limit), p.limit);
      x = rnd<T>(x / (1.f + __expf(-1.702f * x))) * (uu + 1.f);
    } else {
      x = rnd<T>(rnd<T>(x / (1.f + __expf(-x))) * uu);
    }
  }
  return x;
}

template <typename T, bool DUAL>
__global__ void __launch_bounds__(MF_WARPS * 32, 1)
moe_gemm_few_kernel(MoeFewParams p) {
  constexpr int UF = DUAL ? 8 : 16;                  // features of a unit; its second 8 weight rows are the up rows or the next features
  extern __shared__ __align__(16) uint8_t smem[];    // part [2][warp][16 rows][16] fp32 | x [n_pairs][K + pad]
  float* part = reinterpret_cast<float*>(smem);
  T* xs = reinterpret_cast<T*>(smem + 2 * MF_PART * sizeof(float));
  const int ldx = p.K + MF_PAD;
  __shared__ int4 met[MF_PAIRS];                     // the experts' row blocks: (expert, first row, rows); one has a row at least
  __shared__ int s_met;
  pdl_launch_dependents();
  pdl_wait();                                        // the offsets and the grouped rows come from the preceding kernels
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, j = lane & 3;
  if (warp == 0) {
    int n = 0;
    for (int e0 = 0; e0 < p.n_experts; e0 += 32) {
      const int e = e0 + lane, first = e < p.n_experts ? p.offsets[e] : 0;
      const int rows = e < p.n_experts ? p.offsets[e + 1] - first : 0, cnt = (rows + MF_ROWS - 1) / MF_ROWS;
      int at = cnt;                                  // inclusive prefix sum over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, at, o); if (lane >= o) at += v; }
      for (int i = 0; i < cnt; ++i)
        if (n + at - cnt + i < MF_PAIRS) met[n + at - cnt + i] = make_int4(e, first + i * MF_ROWS, min(MF_ROWS, rows - i * MF_ROWS), 0);
      n = min(MF_PAIRS, n + __shfl_sync(0xffffffffu, at, 31));
    }
    if (lane == 0) s_met = n;
  }
  __syncthreads();
  const int per_expert = (p.N + UF - 1) / UF, units = s_met * per_expert, chunks = (p.K + MF_CHUNK - 1) / MF_CHUNK;
  const int mine = (int)blockIdx.x < units ? (units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0, items = mine * chunks;
  const int col_w = warp * 32 * MF_KB + j * 8;       // this lane's first column in a chunk
  const T* W = reinterpret_cast<const T*>(p.W) + (size_t)r * p.K + col_w;
  const size_t second = (size_t)(DUAL ? p.N : 8) * p.K;
  uint4 ring[MF_RING][2][MF_KB];
  // units go round the CTAs; (at, in) is one's place: row block, unit of its expert
  struct Place { int at, in; };
  auto place = [&](Place& q) { while (q.in >= per_expert) { q.in -= per_expert; ++q.at; } };
  auto unit_row = [&](const Place& q) { return W + ((size_t)met[q.at].x * (DUAL ? 2 * p.N : p.N) + q.in * UF) * (size_t)p.K; };
  int req = 0, req_chunk = 0;                        // the next item to request
  Place rq = {0, (int)blockIdx.x};
  place(rq);
  const T* req_row = req < items ? unit_row(rq) : W;
  auto request = [&](uint4 (&w)[2][MF_KB]) {
    const int col = req_chunk * MF_CHUNK;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int b = 0; b < MF_KB; ++b) {
        const bool in = req < items && col_w + col + 32 * b < p.K && (DUAL || x == 0 || rq.in * UF + 8 < p.N);
        w[x][b] = in ? ldg_stream(req_row + x * second + col + 32 * b) : make_uint4(0, 0, 0, 0);
      }
    ++req;
    if (++req_chunk == chunks) {
      req_chunk = 0;
      rq.in += gridDim.x;
      place(rq);
      if (req < items) req_row = unit_row(rq);
    }
  };
#pragma unroll
  for (int i = 0; i < MF_RING; ++i) request(ring[i]);
  {
    const int vecs = p.K / 8;
    const T* A = reinterpret_cast<const T*>(p.A);
    for (int i = threadIdx.x; i < p.n_pairs * vecs; i += MF_WARPS * 32) {
      const int row = i / vecs, c = (i - row * vecs) * 8;
      *reinterpret_cast<uint4*>(xs + (size_t)row * ldx + c) = *reinterpret_cast<const uint4*>(A + (size_t)row * p.lda + c);
    }
  }
  __syncthreads();

  float acc[2][2][4];                                // [weight rows][chain]
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[x][0][e] = acc[x][1][e] = 0.f;
  int chunk = 0, buf = 0;
  Place cur = {0, (int)blockIdx.x};
  place(cur);
  int m0 = items ? met[cur.at].y : 0, rows = items ? met[cur.at].z : 0;
  for (int i0 = 0; i0 < items; i0 += MF_RING) {
#pragma unroll
    for (int d = 0; d < MF_RING; ++d) {
      if (i0 + d >= items) break;                    // the same for the whole CTA
      const int col = chunk * MF_CHUNK + col_w;
      // rows behind the expert's last are another one's: their sums are not used
      const T* x0 = xs + (size_t)min(m0 + r, p.n_pairs - 1) * ldx + col;
      const T* x1 = xs + (size_t)min(m0 + r + 8, p.n_pairs - 1) * ldx + col;
      const bool high = rows > 8;
#pragma unroll
      for (int b = 0; b < MF_KB; ++b) {
        const bool in = col + 32 * b < p.K;
        const uint4 z = make_uint4(0, 0, 0, 0);
        const uint4 a = in ? *reinterpret_cast<const uint4*>(x0 + 32 * b) : z;
        const uint4 c = in && high ? *reinterpret_cast<const uint4*>(x1 + 32 * b) : z;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const uint4& w = ring[d][x][b];
          mma_16816<T>(acc[x][0], a.x, c.x, a.y, c.y, w.x, w.y);
          mma_16816<T>(acc[x][1], a.z, c.z, a.w, c.w, w.z, w.w);
        }
      }
      request(ring[d]);
      if (++chunk < chunks) continue;
      // ---- the unit's sums: acc[x][.][0..1] row r, weight rows 8 x + 2 j and + 1; [2..3] row r + 8
      float* mp = part + (size_t)buf * MF_PART + (size_t)warp * (MF_ROWS * 16);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        float* at = mp + r * 16 + x * 8 + 2 * j;
        *reinterpret_cast<float2*>(at) = make_float2(acc[x][0][0] + acc[x][1][0], acc[x][0][1] + acc[x][1][1]);
        if (high) *reinterpret_cast<float2*>(at + 8 * 16) = make_float2(acc[x][0][2] + acc[x][1][2], acc[x][0][3] + acc[x][1][3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[x][0][e] = acc[x][1][e] = 0.f;
      }
      __syncthreads();                               // the other buffer's readers are through as well
      const int row = threadIdx.x / UF, f = threadIdx.x % UF, n = cur.in * UF + f;
      if (row < rows && n < p.N) {
        const float* at = part + (size_t)buf * MF_PART + row * 16 + f;
        float s = 0.f, u = 0.f;
#pragma unroll
        for (int w = 0; w < MF_WARPS; ++w) {
          s += at[w * (MF_ROWS * 16)];
          if (DUAL) u += at[w * (MF_ROWS * 16) + 8];
        }
        reinterpret_cast<T*>(p.out)[(size_t)(m0 + row) * p.ldo + n] = from_f<T>(moe_few_activate<T, DUAL>(p, s, u));
      }
      buf ^= 1;
      chunk = 0;
      cur.in += gridDim.x;
      place(cur);
      if (i0 + d + 1 < items) { m0 = met[cur.at].y; rows = met[cur.at].z; }
    }
  }
}

template <typename T, bool DUAL>
static int launch_moe_few(const MoeFewParams& p, cudaStream_t st) {
  const size_t smem = sizeof(float) * 2 * MF_PART + sizeof(T) * (size_t)p.n_pairs * (p.K + MF_PAD);
  const long long units = (long long)(p.n_pairs < p.n_experts ? p.n_pairs : p.n_experts) * cdiv(p.N, DUAL ? 8 : 16);
  return launch_pdl("moe_gemm_few", moe_gemm_few_kernel<T, DUAL>, dim3(units < 148 ? (unsigned)units : 148u), dim3(MF_WARPS * 32), smem, st, p);
}

// The rows' columns leave the loads in flight their 90 KB of L1 up to 136 KB, where a row's two products share them, else 128 KB (us,
// weights out of HBM, the tiles and this.  K 2048: gate/up of 24 rows 67 and 45, 32 rows on 8 experts 35 and 29, 48 rows 56 and 91;
// down of 24 rows 40 and 26, 32 rows on 8 experts 16.9 and 17.9; K 1024: gate/up of 64 rows on 2 experts, whose weights are read
// twice each, 20 and 11, down on 16 experts 12.0 and 12.5).
bool moe_gemm_few_wanted(int n_pairs, int K, bool dual) {
  return n_pairs <= MF_PAIRS && 2 * (size_t)n_pairs * (K + MF_PAD) <= (dual ? 136 : 128) * 1024;
}

// 16-bit operands, N and K multiples of 8, 16-byte aligned rows (checked by the caller)
int moe_gemm_few(void* out, int ldo, const void* A, int lda, const void* W, const int32_t* offsets, int n_pairs, int n_experts, int N,
                 int K, int act, float limit, int dtype, cudaStream_t st) {
  const MoeFewParams p = {out, A, W, offsets, ldo, lda, n_pairs, n_experts, N, K, act, limit};
  const bool dual = act == PG_GLU_SILU || act == PG_GLU_CLAMPED;
  if (dtype == PG_BF16) return dual ? launch_moe_few<bf16, true>(p, st) : launch_moe_few<bf16, false>(p, st);
  return dual ? launch_moe_few<f16, true>(p, st) : launch_moe_few<f16, false>(p, st);
}

}  // namespace pg
