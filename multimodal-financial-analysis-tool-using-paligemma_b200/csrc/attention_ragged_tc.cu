// Windowed causal attention with distance bias for ragged token batches on the tcgen05 tensor cores (prompt portions).
//
// The step's tokens are cut on the host into query tiles: up to 128 consecutive tokens of ONE sequence at consecutive
// positions (tile = {first token row, rows, page-table row, first position}).  One CTA = one (tile, head).  The keys a
// tile can see are the positions [max(0, pos0 - window + 1), pos0 + rows - 1] of its sequence, walked page by page
// (key tile = page = 64 keys, fetched by TMA from the paged pools; the append kernel has written the step's own keys
// before this launch).  ONE pass over the key tiles:
//   S(t) = Q K^T (tcgen05.mma, fp32) into one of two TMEM buffers, issued one tile ahead of the softmax;
//   two threads own a query row, 32 of the tile's keys each (their maxima meet in shared memory):
//   z = log2(e) (S * scale - slope_h * (i - j)) - m, masked outside 0 <= i - j < window, in fp32; the row's
//   reference maximum m is raised (and O, sum rescaled, after the products that still add to it) only when a tile exceeds it
//   by more than 2^8; p = exp2(z), row sum from the fp32 values, P rounded to the model dtype and stored over the S
//   columns it came from: O += P V takes P as the TMEM operand and V as an MN-major operand straight from its page.
// What bounds it: the latencies of the softmax's chain (accumulators out of TMEM, the halves' barrier, exponentials, weights into
// TMEM), which four warps on each of an SM's schedulers hide to 40 % of its issue slots; the tiles' products and copies run
// beside it.  So its steps are few: the reference is part of the score's constant, so that the usual tile, which does not raise it,
// subtracts nothing, and distance and scale are two scalar multiply-adds with the key's place as an immediate (in pairs, f32x2, they
// took as many cycles and registers for every constant twice: 231 multiply-add and 213 integer instructions a warp and tile, now
// 184 and 141).  Most tiles lie wholly inside the causal window of all 128 rows and take no masks.  4 prompts of 2048 tokens, 16
// heads of 128, window 1024: 557 us in two passes (row maximum first, S computed twice, P through shared memory, masks on every score),
// 246 in one pass, 219 with the newest pages first, 150 with two threads a row (one: 0.33 instructions a cycle and
// scheduler), 139 with the long tiles first, 141 with exact reciprocals, 124 with the score's constant as above.
// Epilogue: O / sum, times sigmoid(gate), rounded once.  Key width and value width are independent multiples of 64.
// Extensions (pg_attention_ragged_tc_ex): keep_first > 0 keeps the first keep_first positions visible behind the
// window: the window's pages are then followed by those that hold them (as far as they lie before the window's first page).
// sigmoid_weights: p = sigmoid(s + head_bias[h]), no maximum, no sum.  The
// gate may be one value per (token, head); the result is multiplied by out_scale before it is rounded.
// pg_attention_ragged_tc_capped adds a query temperature and a softcap (both fp32, as in attention_ragged.cu; the kernel is
// instantiated with and without the cap).  A capped score is bounded, so its softmax needs no maximum: with a cap of at
// most 40 and bf16 weights (fp32's exponent range) p = exp(s - max(0, sink)).  Head sizes are multiples of 8: the operand
// maps are {column, head, row} tensors, so the 64-column tiles of a narrower head are filled up with zeros by the TMA unit.
// When the value rows are the key rows (or a prefix of them) of ONE pool, P V reads V from the K tile that S = Q K^T has
// just used and nothing is loaded twice.
// Every mbarrier wait is bounded: a wait that gives up sets the error flag, the roles leave their loops, the CTA lets
// its copies land, frees its TMEM and returns.
#include <cmath>

#include "tc_common.cuh"

namespace pg {
namespace tc {

constexpr int WQ = 128;   // query rows per CTA == TMEM lanes
constexpr int WK = 64;    // keys per tile == page size


struct WinParams {
  void* out; int ld_out;
  const void* gate; int ld_gate;
  const int32_t* tiles;          // [n_tiles][4] = {token row0, rows, page-table row, position of row0}
  const int32_t* page_table; int pt_stride;
  int H, kv_group, dim, vdim;
  float scale; int window;
  const float* slopes;
  int* err_flag;
  int keep_first, sigmoid_weights;
  const float* head_bias;
  int gate_per_head;
  float out_scale;
  const float* sink;             // per query head: exp(sink[h]) joins the softmax denominator (NULL: none)
  int chunk;                     // > 0: a key is visible only inside the query's block of `chunk` positions
  const float* out_rot;          // [vdim / 2]: the result is turned back by -position * out_rot[m] (rotated values)
  int out_rot_interleaved;       // pairs (2m, 2m + 1) instead of (m, m + vdim / 2)
  float softcap;                 // > 0: score <- softcap * tanh(score / softcap)
  float temp_coef; int temp_every;   // query temperature 1 + temp_coef * ln(floor((pos + 1) / temp_every) + 1)
  int tied;                      // the value row is (a prefix of) the key row: V is read from the K tile
  int bounded;                   // capped scores that need no maximum: one pass
};

// 1 / (1 + e) for e >= 0, infinity included: one Newton step r (2 - y r) behind the hardware reciprocal, at a quarter of the scale so
// that nothing leaves the range of normal numbers before the last product.  As exact as the rounded division to half a unit
// of fp32 and without its branch: 4 x 2048 tokens, 16 gated heads of 128, 149 us with the division.
__device__ __forceinline__ float inverse_of_1_plus(float e) {
  const float y = fmaf(e, 0.25f, 0.25f);                              // 2^-2 .. 2^126, or infinity
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  r = fmaf(r, fmaf(-fminf(y, 0x1p126f), r, 1.f), r);                  // infinity: 0
  return r * 0.25f;
}

template <typename T, bool CAP>
__global__ void __launch_bounds__(320, 2)
attention_window_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           const __grid_constant__ CUtensorMap map_v, WinParams p) {
  constexpr int FMT = std::is_same<T, bf16>::value ? 1 : 0;
  const int KB = (p.dim + 63) / 64, VB = (p.vdim + 63) / 64;          // 64-column tiles of a head, zero-filled behind it
  const int Q_BYTES = WQ * KB * 128, K_BYTES = WK * KB * 128, V_BYTES = p.tied ? 0 : WK * VB * 128;
  const int O_COL = 2 * WK;                                           // S (and P over it) of even / odd tiles, then O
  const int tmem_cols = (O_COL + VB * 64 <= 256) ? 256 : 512;         // 256 (heads of up to 128): two CTAs share an SM

  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t s_q = base, s_k0 = s_q + Q_BYTES, s_v0 = s_k0 + 2 * K_BYTES, bars = s_v0 + 2 * V_BYTES;
  auto s_k = [&](int bf) { return s_k0 + bf * K_BYTES; };
  auto s_v = [&](int bf) { return p.tied ? s_k(bf) : s_v0 + bf * V_BYTES; };
  // one barrier per buffer: tile t completes phase t >> 1 of barrier t & 1
  const uint32_t bar_q = bars, tmem_slot = bars + 88;
  auto bar_k = [&](int t) { return bars + 8 + 8 * (t & 1); };         // K(t) has landed
  auto bar_v = [&](int t) { return bars + 24 + 8 * (t & 1); };        // V(t) has landed
  auto bar_s = [&](int t) { return bars + 40 + 8 * (t & 1); };        // S(t) is computed
  auto bar_p = [&](int t) { return bars + 56 + 8 * (t & 1); };        // P(t) is stored (and O rescaled)
  auto bar_o = [&](int t) { return bars + 72 + 8 * (t & 1); };        // P(t) V(t) has been added to O
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  __shared__ int s_fail;
  __shared__ float s_half[2][2][WQ];                                  // [tile & 1][half][row]: the halves' maxima, at the end their sums
  volatile int* fail = &s_fail;
  if (threadIdx.x == 0) s_fail = 0;

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x % p.H, kvh = h / p.kv_group;

  if (warp == 1 && lane == 0) {
    mbar_init(bar_q, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_k(i), 1); mbar_init(bar_v(i), 1); mbar_init(bar_s(i), 1); mbar_init(bar_p(i), 256); mbar_init(bar_o(i), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  auto wait = [&](uint32_t bar, int t) { return mbar_wait_lim(bar, (t >> 1) & 1, fail); };
  pdl_wait();  // q, the pools, the tile list and the page table come from the preceding kernels / copies
  // A prompt's later tiles see more keys: the list is walked from its end, the heads of a tile side by side, so that the CTAs
  // of the last, partly filled wave are short ones: 149 -> 139 us (head by head, tiles in list order, SMs were idle 14 % of it).
  const int32_t* tile = p.tiles + 4 * (size_t)((gridDim.x - 1 - blockIdx.x) / p.H);
  const int row0 = tile[0], rows = tile[1], slot = tile[2], pos0 = tile[3];
  const int hi = pos0 + rows - 1;                                        // last key position any row can see
  int lo = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;               // first one
  if (p.chunk > 0) lo = max(lo, pos0 / p.chunk * p.chunk);               // the block of the tile's first row
  const int t_lo = lo / WK;
  // The window's pages from the newest to the oldest, then the pages of the kept first positions that lie before them: a distance
  // bias makes the newest keys the largest, so that a row's reference maximum stands after its own page.  (From the oldest on,
  // it rises by 92 slope per page: heads with slopes above 0.09 rescaled O on every tile, and 556 -> 248 us was all.)
  const int n_keep = (p.keep_first > 0 && p.window > 0) ? min((p.keep_first + WK - 1) / WK, t_lo) : 0;
  const int t_hi = hi / WK, n_win = t_hi - t_lo + 1, n_tiles = n_keep + n_win;
  auto page_of = [&](int t) { return t < n_win ? t_hi - t : t - n_win; };       // key tile -> page of the sequence
  const int32_t* pt_row = p.page_table + (size_t)slot * p.pt_stride;
  const bool sig = p.sigmoid_weights != 0, fixed_max = sig || (CAP && p.bounded);

  if (warp == 0 && lane == 0) {
    // ===================== TMA producer =====================
    mbar_expect_tx(bar_q, Q_BYTES);
    for (int kb = 0; kb < KB; ++kb)
      tma_load_3d(s_q + kb * (WQ * 128), &map_q, bar_q, kb * 64, h, row0);
    for (int t = 0; t < n_tiles; ++t) {
      // the buffers held tile t - 2: its K is free after S(t - 2), its V (or a tied K) after P V of t - 2
      const int row = pt_row[page_of(t)] * WK;
      if (t > 1 && !(p.tied ? wait(bar_o(t), t - 2) : wait(bar_s(t), t - 2))) break;
      mbar_expect_tx(bar_k(t), K_BYTES);
      for (int kb = 0; kb < KB; ++kb)
        tma_load_3d(s_k(t & 1) + kb * (WK * 128), &map_k, bar_k(t), kb * 64, kvh, row);
      if (p.tied) continue;
      if (t > 1 && !wait(bar_o(t), t - 2)) break;
      mbar_expect_tx(bar_v(t), V_BYTES);
      for (int vb = 0; vb < VB; ++vb)
        tma_load_3d(s_v(t & 1) + vb * (WK * 128), &map_v, bar_v(t), vb * 64, kvh, row);
    }
  } else if (warp == 1 && lane == 0) {
    // ===================== MMA issuer =====================
    const uint32_t idesc_s = umma_idesc(FMT, WQ, WK);
    const uint32_t idesc_o = umma_idesc(FMT, WQ, VB * 64) | (1u << 16);            // B (= V) is MN-major
    auto issue_s = [&](int t) {                                      // S(t) = Q K(t)^T
      if (!wait(bar_k(t), t)) return false;
      tc_fence_after();
      for (int ks = 0; ks < (p.dim + 15) / 16; ++ks) {
        const uint32_t off_q = (ks / 4) * (WQ * 128) + (ks % 4) * 32, off_k = (ks / 4) * (WK * 128) + (ks % 4) * 32;
        umma(tmem_base + (t & 1) * WK, umma_desc(s_q + off_q), umma_desc(s_k(t & 1) + off_k), idesc_s, ks > 0 ? 1u : 0u);
      }
      umma_commit(bar_s(t));
      return true;
    };
    bool ok = mbar_wait_lim(bar_q, 0, fail) && issue_s(0);
    for (int t = 0; ok && t < n_tiles; ++t) {
      if (t + 1 < n_tiles) {                                         // P(t - 1) lies where S(t + 1) goes
        if (t > 0 && !wait(bar_o(t - 1), t - 1)) break;
        if (!issue_s(t + 1)) break;
      }
      if (!wait(bar_p(t), t)) break;
      if (!p.tied && !wait(bar_v(t), t)) break;
      tc_fence_after();
      for (int ks = 0; ks < WK / 16; ++ks)                           // O += P(t) V(t)
        umma_ts(tmem_base + O_COL, tmem_base + (t & 1) * WK + ks * 8, umma_desc_mn(s_v(t & 1) + ks * 2048, WK * 128), idesc_o,
                (t > 0 || ks > 0) ? 1u : 0u);
      umma_commit(bar_o(t));
    }
  } else if (warp >= 2) {
    // ===================== softmax + epilogue: two threads per query row, 32 of a tile's keys each =====================
    // A wait that gave up leaves the loops running (every later wait returns at once): the two halves meet at barriers.
    const int qw = warp & 3, r = qw * 32 + lane, hf = (warp - 2) >> 2;   // TMEM lane quarter = warp & 3
    auto meet = [&] {                                              // the two warps of these 32 rows
      __syncwarp();
      asm volatile("bar.sync %0, 64;" ::"r"(1 + qw) : "memory");
    };
    constexpr int HK = WK / 2;
    const uint32_t t_row = tmem_base + ((uint32_t)(qw * 32) << 16);
    const int i = pos0 + r;                                        // this row's position
    const float slope = (p.slopes ? p.slopes[h] : 0.f) * LOG2E_F, hbias = (p.head_bias ? p.head_bias[h] : 0.f) * LOG2E_F;
    // the first position that this row sees but for kept ones: its window's, and its block's
    const int first = max(p.chunk > 0 ? i / p.chunk * p.chunk : 0, p.window > 0 ? i - p.window + 1 : 0);
    const int blk_last = p.chunk > 0 ? (pos0 + WQ - 1) / p.chunk * p.chunk : 0;
    float m = -INFINITY, l = 0.f;                                  // m in units of log2
    if (CAP && p.bounded) m = (p.sink ? fmaxf(p.sink[h], 0.f) : 0.f) * LOG2E_F;  // any value near the scores does: they are bounded
    if (sig) m = 0.f;
    float qscale = p.scale;
    if (CAP && p.temp_every > 0) qscale *= 1.f + p.temp_coef * logf((float)((i + 1) / p.temp_every + 1));
    const float cap_in = CAP ? 2.f * qscale / p.softcap : 0.f, cap_out = 2.f * p.softcap;
    const float qs2 = qscale * LOG2E_F;
    bool ok = true;
    for (int t = 0; t < n_tiles; ++t) {
      ok = wait(bar_s(t), t) && ok;
      tc_fence_after();
      const int page0 = page_of(t) * WK, j0 = page0 + hf * HK;
      float s[HK];
      tmem_ld32(t_row + (t & 1) * WK + hf * HK, s);
      tmem_ld_wait();
      if (CAP) {       // cap * tanh(z / cap) = cap - 2 cap / (exp(2 z / cap) + 1): absolute error a few 1e-7 of the cap
#pragma unroll
        for (int jj = 0; jj < HK; ++jj) s[jj] = (p.softcap - __fdividef(cap_out, __expf(s[jj] * cap_in) + 1.f)) * LOG2E_F;
      }
      // slope (j - i) + bias - the row's reference, from its value at the thread's first key
      const float ref = m == -INFINITY ? 0.f : m;                  // a row that has seen no key yet
      const float z0 = fmaf(slope, (float)(j0 - i), hbias - ref);
#pragma unroll
      for (int jj = 0; jj < HK; ++jj) {
        const float z = fmaf(slope, (float)jj, z0);
        s[jj] = CAP ? s[jj] + z : fmaf(s[jj], qs2, z);
      }
      // whole tiles that every row sees need no masks
      const bool full = page0 + WK - 1 <= pos0 && page0 >= blk_last &&
                        (p.window <= 0 || pos0 + WQ - 1 - page0 < p.window || page0 + WK <= p.keep_first);
      if (!full) {                                                 // visible: first <= j <= i, or a kept first position up to i
        const unsigned span = (unsigned)(i - first), at = (unsigned)(j0 - first);
        const int kept = min(p.keep_first, i + 1) - j0;
#pragma unroll
        for (int jj = 0; jj < HK; ++jj) s[jj] = (at + jj <= span || jj < kept) ? s[jj] : -INFINITY;
      }
      float top = -INFINITY;
      if (!fixed_max) {
        float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int jj = 4; jj < HK; ++jj) mx[jj & 3] = fmaxf(mx[jj & 3], s[jj]);
        top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        s_half[t & 1][hf][r] = top;
      }
      meet();                                                      // both have read their scores: P may take S's columns
      if (!fixed_max) {
        top = fmaxf(top, s_half[t & 1][hf ^ 1][r]);                // the same in both threads, and so is every decision below
        if (__any_sync(0xffffffffu, top > (m == -INFINITY ? -INFINITY : MAX_RAISE))) {   // m == -inf: any visible key raises it
          const float m_new = fmaxf(m, top + ref);
          if (t > 0) {
            const float corr = m_new == m ? 1.f : exp2_approx(m - m_new);
            l *= corr;
            ok = wait(bar_o(t - 1), t - 1) && ok;                    // nothing adds to O until this tile's P is handed over
            tc_fence_after();
#pragma unroll 1
            for (int c = hf; c < VB * 4; c += 2) {
              float o[16];
              tmem_ld16(t_row + O_COL + c * 16, o);
              tmem_ld_wait();
#pragma unroll
              for (int jj = 0; jj < 16; ++jj) o[jj] *= corr;
              tmem_st16(t_row + O_COL + c * 16, reinterpret_cast<const uint32_t*>(o));
            }
          }
          m = m_new;
          const float up = (m == -INFINITY ? 0.f : m) - ref;
#pragma unroll
          for (int jj = 0; jj < HK; ++jj) s[jj] -= up;
        }
      }
      if (sig) {
#pragma unroll
        for (int jj = 0; jj < HK; ++jj) s[jj] = inverse_of_1_plus(exp2_approx(-s[jj]));   // exp2(+inf) -> weight 0 when masked
      } else {
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int jj = 0; jj < HK; ++jj) {
          s[jj] = exp2_approx(s[jj]);
          sum[jj & 3] += s[jj];
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      }
      uint32_t pk[HK / 2];
#pragma unroll
      for (int jj = 0; jj < HK / 2; ++jj) pk[jj] = pack_pair<T>(s[2 * jj], s[2 * jj + 1]);
      tmem_st16(t_row + (t & 1) * WK + hf * (HK / 2), pk);         // P takes the first 32 of the row's S columns
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar_p(t));
    }
    s_half[n_tiles & 1][hf][r] = l;
    meet();
    l = s_half[n_tiles & 1][0][r] + s_half[n_tiles & 1][1][r];
    if (__all_sync(0xffffffffu, wait(bar_o(n_tiles - 1), n_tiles - 1) && ok)) {   // the loads below take the whole warp
      tc_fence_after();
      if (p.sink && !sig) l += exp2_approx(p.sink[h] * LOG2E_F - m);   // a logit without key or value, counted once
      float inv = (sig ? 1.f : 1.f / l) * p.out_scale;
      const size_t trow = (size_t)row0 + r;
      T* orow = reinterpret_cast<T*>(p.out) + trow * p.ld_out + (size_t)h * p.vdim;
      const T* grow = (p.gate && !p.gate_per_head) ? reinterpret_cast<const T*>(p.gate) + trow * p.ld_gate + (size_t)h * p.vdim : nullptr;
      if (p.gate && p.gate_per_head && r < rows)
        inv *= 1.f / (1.f + __expf(-to_f<T>(reinterpret_cast<const T*>(p.gate)[trow * p.ld_gate + h])));
      auto store32 = [&](int c, const float* o) {                  // 32 finished columns of this row: gate, round, store
        if (r >= rows) return;
#pragma unroll
        for (int q0 = 0; q0 < 32; q0 += 8) {
          if (c * 32 + q0 >= p.vdim) break;                        // vdim is a multiple of 8
          float w[8], gt[8];
          if (grow) unpack<T>(*reinterpret_cast<const uint4*>(grow + c * 32 + q0), gt);
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) {
            float v = o[q0 + jj];
            if (grow) v *= inverse_of_1_plus(__expf(-gt[jj]));
            w[jj] = v;
          }
          *reinterpret_cast<uint4*>(orow + c * 32 + q0) = pack<T>(w);
        }
      };
      const float fpos = (float)i;
      if (!p.out_rot) {
#pragma unroll 1
        for (int c = hf; c * 32 < p.vdim; c += 2) {
          float o[32];
          tmem_ld32(t_row + O_COL + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) o[jj] *= inv;
          store32(c, o);
        }
      } else if (p.out_rot_interleaved) {                          // pairs of neighbours: both halves in one load
#pragma unroll 1
        for (int c = hf; c * 32 < p.vdim; c += 2) {
          float o[32];
          tmem_ld32(t_row + O_COL + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float sn, cs;
            sincosf(-fpos * p.out_rot[c * 16 + k], &sn, &cs);
            const float u = o[2 * k] * inv, v = o[2 * k + 1] * inv;
            o[2 * k] = u * cs - v * sn;
            o[2 * k + 1] = v * cs + u * sn;
          }
          store32(c, o);
        }
      } else {                                                     // column m with m + vdim / 2 (vdim is a multiple of 64)
        const int hc = p.vdim / 64;
#pragma unroll 1
        for (int c = hf; c < hc; c += 2) {
          float a[32], b[32];
          tmem_ld32(t_row + O_COL + c * 32, a);
          tmem_ld32(t_row + O_COL + (hc + c) * 32, b);
          tmem_ld_wait();
#pragma unroll
          for (int jj = 0; jj < 32; ++jj) {
            float sn, cs;
            sincosf(-fpos * p.out_rot[c * 32 + jj], &sn, &cs);
            const float u = a[jj] * inv, v = b[jj] * inv;
            a[jj] = u * cs - v * sn;
            b[jj] = v * cs + u * sn;
          }
          store32(c, a);
          store32(hc + c, b);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (s_fail) {  // let copies and MMAs that are still in flight finish before the shared memory and TMEM go away
    for (int k = 0; k < 2000; ++k) __nanosleep(1000);
    if (threadIdx.x == 0 && p.err_flag) *p.err_flag = 2;
    __syncthreads();
  }
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

}  // namespace tc
}  // namespace pg

using namespace pg;

extern "C" int pg_attention_ragged_tc_ok(int dim, int vdim, int page_size, int ld_q, int ld_out, int ld_gate, int dtype) {
  static const int enabled = env_int("PG_RAGGED_ATTN_TC", 1);
  if (!enabled || (dtype != PG_BF16 && dtype != PG_F16) || page_size != tc::WK) return 0;
  if (dim % 64 || vdim % 64 || dim > 256 || vdim > 256 || ld_q % 8 || ld_out % 8 || ld_gate % 8) return 0;
  return tc::encode_fn() != nullptr ? 1 : 0;
}

extern "C" int pg_attention_ragged_tc_ok8(int dim, int vdim, int page_size, int ld_q, int ld_out, int ld_gate, int dtype) {
  static const int enabled = env_int("PG_RAGGED_ATTN_TC", 1);
  if (!enabled || (dtype != PG_BF16 && dtype != PG_F16) || page_size != tc::WK) return 0;
  if (dim % 8 || vdim % 8 || dim > 256 || vdim > 256 || ld_q % 8 || ld_out % 8 || ld_gate % 8) return 0;
  return tc::encode_fn() != nullptr ? 1 : 0;
}

extern "C" int pg_attention_ragged_tc_sink(void* out, int ld_out, const void* q, int ld_q, const void* gate, int ld_gate,
                                           int gate_per_head, const void* k_pool, int ld_k, const void* v_pool, int ld_v,
                                           long long pool_rows, const int32_t* page_table, int pt_stride, int page_size,
                                           const int32_t* tiles, int n_tiles, int n_tokens, int n_heads, int n_kv_heads,
                                           int dim, int vdim, float scale, int window, int keep_first,
                                           const float* slopes, int sigmoid_weights, const float* head_bias,
                                           const float* sink, float out_scale, int* err_flag, int dtype, void* stream) {
  return pg_attention_ragged_tc_masked(out, ld_out, q, ld_q, gate, ld_gate, gate_per_head, k_pool, ld_k, v_pool, ld_v, pool_rows,
                                       page_table, pt_stride, page_size, tiles, n_tiles, n_tokens, n_heads, n_kv_heads, dim,
                                       vdim, scale, window, keep_first, 0, slopes, sigmoid_weights, head_bias, sink, nullptr, 0,
                                       out_scale, err_flag, dtype, stream);
}

extern "C" int pg_attention_ragged_tc_masked(void* out, int ld_out, const void* q, int ld_q, const void* gate, int ld_gate,
                                             int gate_per_head, const void* k_pool, int ld_k, const void* v_pool, int ld_v,
                                             long long pool_rows, const int32_t* page_table, int pt_stride, int page_size,
                                             const int32_t* tiles, int n_tiles, int n_tokens, int n_heads, int n_kv_heads,
                                             int dim, int vdim, float scale, int window, int keep_first, int chunk,
                                             const float* slopes, int sigmoid_weights, const float* head_bias,
                                             const float* sink, const float* out_rot, int out_rot_interleaved,
                                             float out_scale, int* err_flag, int dtype, void* stream) {
  return pg_attention_ragged_tc_capped(out, ld_out, q, ld_q, gate, ld_gate, gate_per_head, k_pool, ld_k, v_pool, ld_v, pool_rows,
                                       page_table, pt_stride, page_size, tiles, n_tiles, n_tokens, n_heads, n_kv_heads, dim,
                                       vdim, scale, window, keep_first, chunk, slopes, sigmoid_weights, head_bias, sink, 0.f,
                                       0.f, 0, out_rot, out_rot_interleaved, out_scale, err_flag, dtype, stream);
}

extern "C" int pg_attention_ragged_tc_capped(void* out, int ld_out, const void* q, int ld_q, const void* gate, int ld_gate,
                                             int gate_per_head, const void* k_pool, int ld_k, const void* v_pool, int ld_v,
                                             long long pool_rows, const int32_t* page_table, int pt_stride, int page_size,
                                             const int32_t* tiles, int n_tiles, int n_tokens, int n_heads, int n_kv_heads,
                                             int dim, int vdim, float scale, int window, int keep_first, int chunk,
                                             const float* slopes, int sigmoid_weights, const float* head_bias,
                                             const float* sink, float softcap, float temp_coef, int temp_every,
                                             const float* out_rot, int out_rot_interleaved, float out_scale, int* err_flag,
                                             int dtype, void* stream) {
  if (n_tiles <= 0) return PG_OK;
  PG_REQUIRE(chunk >= 0 && (chunk == 0 || keep_first == 0), "attention_ragged_tc: blocks of %d positions with %d kept first ones",
             chunk, keep_first);
  if (ld_k <= 0) ld_k = n_kv_heads * dim;
  if (ld_v <= 0) ld_v = n_kv_heads * vdim;
  PG_REQUIRE(ld_k >= n_kv_heads * dim && ld_v >= n_kv_heads * vdim && ld_k % 8 == 0 && ld_v % 8 == 0,
             "attention_ragged_tc: pool rows of %d / %d elements", ld_k, ld_v);
  PG_REQUIRE(pg_attention_ragged_tc_ok8(dim, vdim, page_size, ld_q, ld_out, (gate && !gate_per_head) ? ld_gate : 8, dtype),
             "attention_ragged_tc: unsupported problem (dim %d vdim %d page %d dtype %d)", dim, vdim, page_size, dtype);
  PG_REQUIRE(!out_rot || vdim % 64 == 0, "attention_ragged_tc: values of %d columns that are turned back", vdim);
  PG_REQUIRE(softcap >= 0.f && temp_every >= 0 && (temp_every == 0 || softcap > 0.f),
             "attention_ragged_tc: softcap %g, temperature steps of %d (a temperature needs a cap here)", (double)softcap, temp_every);
  PG_REQUIRE(n_heads % n_kv_heads == 0, "attention_ragged_tc: heads %d / kv heads %d", n_heads, n_kv_heads);
  PG_REQUIRE(((uintptr_t)q % 16) == 0 && ((uintptr_t)out % 16) == 0 && (gate_per_head || ((uintptr_t)gate % 16) == 0) &&
                 ((uintptr_t)k_pool % 16) == 0 && ((uintptr_t)v_pool % 16) == 0,
             "attention_ragged_tc: operands must be 16-byte aligned");
  const bool bf = dtype == PG_BF16;
  CUtensorMap mq, mk, mv;
  PG_REQUIRE(tc::make_map_heads(&mq, q, n_tokens, n_heads, dim, ld_q, tc::WQ, bf) &&
                 tc::make_map_heads(&mk, k_pool, pool_rows, n_kv_heads, dim, ld_k, tc::WK, bf) &&
                 tc::make_map_heads(&mv, v_pool, pool_rows, n_kv_heads, vdim, ld_v, tc::WK, bf),
             "attention_ragged_tc: cuTensorMapEncodeTiled failed");
  const int tied = (k_pool == v_pool && ld_k == ld_v && (dim == vdim || (n_kv_heads == 1 && vdim < dim))) ? 1 : 0;
  const int bounded = (bf && softcap > 0.f && softcap <= 40.f && !sigmoid_weights && !slopes && !head_bias) ? 1 : 0;
  tc::WinParams p = {out, ld_out, gate, ld_gate, tiles, page_table, pt_stride, n_heads, n_heads / n_kv_heads, dim, vdim,
                     scale, window, slopes, err_flag, keep_first, sigmoid_weights ? 1 : 0, head_bias,
                     gate_per_head ? 1 : 0, out_scale, sink, chunk, out_rot, out_rot_interleaved ? 1 : 0, softcap, temp_coef,
                     temp_every, tied, bounded};
  const int kb = cdiv(dim, 64), vb = cdiv(vdim, 64);
  const size_t smem = 1024 + (size_t)tc::WQ * kb * 128 + 2 * (size_t)tc::WK * kb * 128 +
                      (tied ? 0 : 2 * (size_t)tc::WK * vb * 128) + 88 + 8;
  cudaStream_t st = (cudaStream_t)stream;
  PG_REQUIRE(n_heads <= 65535 && (long long)n_tiles * n_heads < (1ll << 31), "attention_ragged_tc: %d tiles of %d heads", n_tiles, n_heads);
  dim3 grid((unsigned)n_tiles * n_heads);
  auto run = [&](auto kern) -> int {
    PG_REQUIRE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess,
               "attention_ragged_tc: cannot reserve %zu B of shared memory", smem);
    return launch_tc("attention_ragged_tc", kern, grid, dim3(320), smem, 1, false, st, mq, mk, mv, p);
  };
  if (softcap > 0.f) return bf ? run(tc::attention_window_tc_kernel<bf16, true>) : run(tc::attention_window_tc_kernel<f16, true>);
  return bf ? run(tc::attention_window_tc_kernel<bf16, false>) : run(tc::attention_window_tc_kernel<f16, false>);
}

extern "C" int pg_attention_ragged_tc_ex(void* out, int ld_out, const void* q, int ld_q, const void* gate, int ld_gate,
                                         int gate_per_head, const void* k_pool, const void* v_pool, long long pool_rows,
                                         const int32_t* page_table, int pt_stride, int page_size, const int32_t* tiles,
                                         int n_tiles, int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim,
                                         float scale, int window, int keep_first, const float* slopes,
                                         int sigmoid_weights, const float* head_bias, float out_scale, int* err_flag,
                                         int dtype, void* stream) {
  return pg_attention_ragged_tc_sink(out, ld_out, q, ld_q, gate, ld_gate, gate_per_head, k_pool, 0, v_pool, 0, pool_rows,
                                     page_table, pt_stride, page_size, tiles, n_tiles, n_tokens, n_heads, n_kv_heads, dim,
                                     vdim, scale, window, keep_first, slopes, sigmoid_weights, head_bias, nullptr, out_scale,
                                     err_flag, dtype, stream);
}

extern "C" int pg_attention_ragged_tc(void* out, int ld_out, const void* q, int ld_q, const void* gate, int ld_gate,
                                      const void* k_pool, const void* v_pool, long long pool_rows,
                                      const int32_t* page_table, int pt_stride, int page_size, const int32_t* tiles,
                                      int n_tiles, int n_tokens, int n_heads, int n_kv_heads, int dim, int vdim,
                                      float scale, int window, const float* slopes, int* err_flag, int dtype,
                                      void* stream) {
  return pg_attention_ragged_tc_ex(out, ld_out, q, ld_q, gate, ld_gate, 0, k_pool, v_pool, pool_rows, page_table, pt_stride,
                                   page_size, tiles, n_tiles, n_tokens, n_heads, n_kv_heads, dim, vdim, scale, window, 0,
                                   slopes, 0, nullptr, 1.f, err_flag, dtype, stream);
}
