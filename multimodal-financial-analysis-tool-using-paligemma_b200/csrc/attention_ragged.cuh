// Parameters and key order of the attention over ragged token batches (attention_ragged.cu, attention_ragged_mma.cu).
#pragma once
#include "common.cuh"

namespace pg {

struct RagAttnParams {
  void* out; int ld_out;
  const void* q; int ld_q;
  const void* gate; int ld_gate;
  const void* k_pool; const void* v_pool;
  const int32_t* page_table; int pt_stride; int page_size;
  const int32_t* tok_slot; const int32_t* tok_pos;
  int n_tokens, H, G, dim, vdim;
  float scale; int window;
  const float* slopes;
  int keep_first;                // positions < keep_first stay visible behind the window
  int sigmoid_weights;           // 0: softmax over the visible keys; 1: weight = sigmoid(score + head_bias[h])
  const float* head_bias;        // per query head, added to the score (NULL: none)
  int gate_per_head;             // 0: gate[t][h * vdim + c]; 1: gate[t][h]
  float out_scale;
  int ld_k, ld_v;                // elements between the rows of the key / value pool (>= G * dim, G * vdim)
  const float* sink;             // per query head: exp(sink[h]) joins the softmax denominator (no key, no value)
  int chunk;                     // > 0: a key is visible only inside the query's block of `chunk` positions
  const float* out_rot;          // [vdim / 2]: the result is turned back by -position * out_rot[m] (rotated values)
  int out_rot_interleaved;       // pairs (2m, 2m + 1) instead of (m, m + vdim / 2)
  float softcap;                 // > 0: score <- softcap * tanh(score / softcap)
  float temp_coef; int temp_every;   // query temperature 1 + temp_coef * ln(floor((pos + 1) / temp_every) + 1)
};

// The factor of q . k for a query at position pos.
__device__ __forceinline__ float query_scale(const RagAttnParams& p, int pos) {
  return p.temp_every > 0 ? p.scale * (1.f + p.temp_coef * logf((float)((pos + 1) / p.temp_every + 1))) : p.scale;
}
__device__ __forceinline__ float capped(const RagAttnParams& p, float s) {
  return p.softcap > 0.f ? p.softcap * tanhf(s / p.softcap) : s;
}

// The visible keys of a token at position pos as one list: n_keep kept first positions, then [lo, pos].
struct KeyRange {
  int lo, n_keep, count;
  __device__ __forceinline__ KeyRange(int pos, int window, int keep_first, int chunk = 0) {
    lo = window > 0 ? max(0, pos - window + 1) : 0;
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);   // blocks are counted from position 0 of the sequence
    n_keep = min(max(keep_first, 0), lo);
    count = n_keep + pos - lo + 1;
  }
  __device__ __forceinline__ int key(int v) const { return v < n_keep ? v : lo + (v - n_keep); }
};

// attention_ragged_mma.cu: 16-bit problems whose heads fit its fragments; false: the other kernels take it
bool attention_ragged_mma_wanted(const RagAttnParams& p, int dtype);
int attention_ragged_mma(const RagAttnParams& p, int dtype, cudaStream_t st);

}  // namespace pg
