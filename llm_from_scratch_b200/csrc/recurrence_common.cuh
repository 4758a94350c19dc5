// Pieces shared by the gated recurrence's kernels: arguments and the gates of a channel.
#pragma once

#include "sequences.cuh"

namespace b200 {

struct RecArgs {
  const void* q;
  const void* f;
  const void* v;
  int64_t stride;            // elements between tokens, the same for q / f / v (views of one projection)
  const float* f_bias;       // [H, dk]
  const float* lower;        // [H, dk]
  const float* norm_w;       // [dv]
  float eps;
  float* state;              // [slots, H, dk, dv]
  const int64_t* slots;      // [n], < 0: skip the sequence
  int64_t num_slots;
  const int32_t* cu_q;       // [n + 1], or null: one token per sequence
  const int32_t* cu_k;       // [n + 1] with cu_q
  const int64_t* ctx_lens;   // [n] without cu_q: context length including the new token
  void* out;                 // [T, H, dv]
  int H, dk, dv;
  int32_t* status;
};

// forget gate and write gate of one channel
__device__ __forceinline__ void gates(float z, float lower, float* f, float* k) {
  const float open = 1.f - lower;
  float s, n;
  sigmoids(z, &s, &n);
  *f = lower + open * s;
  *k = open * n;
}

struct ScanArgs {
  float* seg_state;          // [segments, H, dk, dv]  pass 1: P, after pass 2: entry state
  float* seg_decay;          // [segments, H, dk]      pass 1: D
  int n, seg_len;
  bool async;                // 16-byte copies are possible
};

// prompts and portions on tensor cores (recurrence_chunk.cu): bf16, dk = dv = 64 or 128, 16-byte aligned rows
inline bool recurrence_chunk_shape(int dk, int dv) { return dk == dv && (dk == 64 || dk == 128); }
bool recurrence_chunk_pays(int n, int64_t total_tokens, int max_seqlen_q, int H, int D);
int recurrence_chunk_seg_len(int64_t total_tokens, int max_seqlen_q, int H);
int recurrence_chunk_launch(const RecArgs& a, const ScanArgs& sc, int64_t segments, bool chained, cudaStream_t s);

// entry states of all segments (pass 2)
int recurrence_chain_launch(const RecArgs& a, const ScanArgs& sc, cudaStream_t s);

}  // namespace b200
