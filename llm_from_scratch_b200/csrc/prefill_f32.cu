// Ragged causal prefill attention in fp32: head sizes 32, 64 and 128, packed or paged keys, optional sinks.
//
// Bound by the fp32 pipe (4 d FMAs per visible (query, key, head) triple; no matrix unit multiplies fp32 by fp32), so the
// kernel is a register-tiled product: a CTA holds RM * 16 rows of one KV head, a row being a (query token, query head) pair,
// so that the heads of a group share every K and V tile and the causal diagonal crosses RM * 16 / G tokens only.  A thread
// owns RM rows x BN / 8 keys of the scores and RM rows x D / 8 columns of the output.  K and V tiles have one buffer each: V
// arrives under the scores, the next K under softmax and P V; two to four CTAs of an SM fill each other's waits.  The eight
// lanes of a row exchange maxima by shuffles and probabilities through rows of shared memory that only their warp touches.
//
// Measured on 8 prompts of 64 to 1024 tokens, 16/4 heads x 64: 340 us (the general kernel, a warp per row that reads every
// key for itself: 6,620 us), half of the fp32 pipe's rate.  Scores as one chain of 64 products took 315 us, but their error
// against 64 bits was 3.1e-7 (the general kernel's: 3.0e-7; with chains of 32: 2.6e-7).  Row tiles of 128 (RM = 8) were no
// faster; in the general grid's order, one sequence after the other, the kernel took 80 us more.
#include "sequences.cuh"

namespace b200 {
namespace {

struct PrefillF32Args {
  const float* q;
  const float* k;            // packed keys / values, or the pools with bt
  const float* v;
  float* out;
  int64_t q_stride, k_stride, v_stride;  // token strides, elements
  const int32_t* cu_q;
  const int32_t* cu_k;
  int num_seqs, Hq, Hkv;
  float scale_log2;
  const int32_t* bt;         // null: packed
  int64_t bt_stride;
  int bs;
  int64_t num_blocks;
  const float* sink;         // [Hq] or null
  int32_t* status;
};

constexpr int kThreads = 128;      // 16 row groups x 8 key / column groups

// keys per tile: scores and outputs of a thread stay within the register file
__host__ __device__ constexpr int tile_keys(int D) { return D == 128 ? 32 : 64; }
__host__ __device__ constexpr size_t smem_bytes(int D, int RM) {
  const int bm = RM * 16, bn = tile_keys(D);
  return sizeof(float) * (static_cast<size_t>(bm) * (D + 4) + bn * (D + 4) + bn * D + bm * (bn + 8)) + bn * sizeof(int);
}

template <int D, int RM>
__global__ void __launch_bounds__(kThreads, RM == 2 ? 4 : D == 128 ? 2 : 3) prefill_f32_kernel(const PrefillF32Args a) {
  constexpr int BM = RM * 16, BN = tile_keys(D), CN = BN / 8, OC = D / 8;
  constexpr int QS = D + 4, PS = BN + 8;       // row strides that spread the rows of a warp over the banks
  extern __shared__ __align__(16) float sm[];
  float* sq = sm;                              // [BM][QS]
  float* sk = sq + BM * QS;                    // [BN][QS]
  float* sv = sk + BN * QS;                    // [BN][D]
  float* sp = sv + BN * D;                     // [BM][PS]
  int* skip = reinterpret_cast<int*>(sp + BM * PS);   // [BN] keys whose block is outside the pool

  // Row tiles from the highest to the lowest, all sequences and heads of one before the next: a tile's work grows with
  // its number, so the longest CTAs start first (with one sequence after the other the last one's ran alone at the end).
  const int per_tile = a.num_seqs * a.Hkv, tile = (gridDim.x - 1 - blockIdx.x) / per_tile, pair = blockIdx.x % per_tile;
  const int s = pair % a.num_seqs, kvh = pair / a.num_seqs, G = a.Hq / a.Hkv;
  const int q0 = a.cu_q[s], q_len = a.cu_q[s + 1] - q0;
  const int k0 = a.cu_k[s], k_len = a.cu_k[s + 1] - k0;
  const int64_t rows = static_cast<int64_t>(q_len) * G, row0 = static_cast<int64_t>(tile) * BM;
  if (row0 >= rows) return;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int live = static_cast<int>(rows - row0 < BM ? rows - row0 : BM);
  const int before = k_len - q_len;            // keys ahead of the first query's own
  // keys that some row of the tile sees, and that all of them see
  const int most = min(before + static_cast<int>((row0 + live - 1) / G) + 1, k_len);
  const int least = before + static_cast<int>(row0 / G) + 1;
  const int table_keys = a.bt ? static_cast<int>(min(a.bt_stride * a.bs, static_cast<int64_t>(k_len))) : k_len;
  if (a.bt && table_keys < most && tid == 0) report(a.status, B200_ERR_BOUNDS);

  for (int i = tid; i < BM * (D / 4); i += kThreads) {
    const int r = i / (D / 4), c = i % (D / 4);
    const int64_t row = row0 + (r < live ? r : 0);
    const int64_t off = (q0 + row / G) * a.q_stride + static_cast<int64_t>(kvh * G + row % G) * D + c * 4;
    cp_async16(smem_u32(sq + r * QS + c * 4), a.q + off, r < live ? 16 : 0);
  }

  // 16-byte pieces of a tile: a row's pieces lie in consecutive lanes
  auto load = [&](const float* src, int64_t stride, float* dst, int dst_row, int j0, bool mark) {
#pragma unroll 4
    for (int i = tid; i < BN * (D / 4); i += kThreads) {
      const int r = i / (D / 4), c = i % (D / 4), j = j0 + r;
      int64_t off = 0;
      bool ok = j < most;
      if (a.bt == nullptr) {
        off = (k0 + static_cast<int64_t>(j)) * stride + static_cast<int64_t>(kvh) * D;
      } else {
        ok = ok && j < table_keys;
        const int64_t id = ok ? a.bt[static_cast<int64_t>(s) * a.bt_stride + j / a.bs] : 0;
        if (static_cast<uint64_t>(id) >= static_cast<uint64_t>(a.num_blocks)) {
          report(a.status, B200_ERR_BOUNDS);
          ok = false;
        }
        off = ((id * a.bs + j % a.bs) * a.Hkv + kvh) * D;
        if (mark && c == 0) skip[r] = !ok;
      }
      cp_async16(smem_u32(dst + r * dst_row + c * 4), ok ? src + off + c * 4 : src, ok ? 16 : 0);
    }
    cp_async_commit();
  };

  int nkeys[RM];                               // keys this thread's rows see
  f32x2 o[RM][OC / 2];
  float m[RM], l[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int r = ty + 16 * i;
    nkeys[i] = r < live ? before + static_cast<int>((row0 + r) / G) + 1 : 0;
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < OC / 2; ++c) o[i][c] = 0;
  }

  load(a.k, a.k_stride, sk, QS, 0, true);
  for (int j0 = 0; j0 < most; j0 += BN) {
    load(a.v, a.v_stride, sv, D, j0, false);
    cp_async_wait<1>();
    __syncthreads();
    // ---- scores ----
    float x[RM][CN];
    {
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) x[i][j] = 0.f;
      // chains of 32 channels: no longer than the general kernel's sums, so no less exact
#pragma unroll 1
      for (int d0 = 0; d0 < D; d0 += 32) {
        float part[RM][CN];
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int j = 0; j < CN; ++j) part[i][j] = 0.f;
#pragma unroll 8
        for (int d = d0; d < d0 + 32; d += 2) {
          float2 qv[RM], kv[CN];
#pragma unroll
          for (int i = 0; i < RM; ++i) qv[i] = *reinterpret_cast<const float2*>(sq + (ty + 16 * i) * QS + d);
#pragma unroll
          for (int j = 0; j < CN; ++j) kv[j] = *reinterpret_cast<const float2*>(sk + (tx + 8 * j) * QS + d);
#pragma unroll
          for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < CN; ++j) part[i][j] = fmaf(qv[i].y, kv[j].y, fmaf(qv[i].x, kv[j].x, part[i][j]));
        }
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int j = 0; j < CN; ++j) x[i][j] += part[i][j];
      }
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) x[i][j] *= a.scale_log2;
    }
    const bool border = j0 + BN > least;
    if (border) {
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j)
          if (j0 + tx + 8 * j >= nkeys[i]) x[i][j] = -INFINITY;
    }
    if (a.bt) {
#pragma unroll
      for (int j = 0; j < CN; ++j)
        if (skip[tx + 8 * j]) {
#pragma unroll
          for (int i = 0; i < RM; ++i) x[i][j] = -INFINITY;
        }
    }
    // ---- online softmax ----
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      float mx = x[i][0];
#pragma unroll
      for (int j = 1; j < CN; ++j) mx = fmaxf(mx, x[i][j]);
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float mn = fmaxf(m[i], mx), ref = mn == -INFINITY ? 0.f : mn;     // no key yet: weights 0
      const float al = exp2f(m[i] - ref);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < CN; ++j) {
        const float p = exp2f(x[i][j] - ref);
        sum += p;
        sp[(ty + 16 * i) * PS + tx + 8 * j] = p;
      }
      m[i] = mn;
      l[i] = l[i] * al + sum;
      const f32x2 al2 = pack2(al, al);
#pragma unroll
      for (int c = 0; c < OC / 2; ++c) o[i][c] = mul2(o[i][c], al2);
    }
    cp_async_wait<0>();
    __syncthreads();
    if (j0 + BN < most) load(a.k, a.k_stride, sk, QS, j0 + BN, true);
    // A weight of 0 must not meet an infinity or NaN of a value that its row does not see: tiles that some row sees only a
    // part of are searched for one, and then take the products row by row.
    bool careful = false;
    if (border) {
      bool odd = false;
      for (int i = tid; i < BN * D; i += kThreads) odd |= !isfinite(sv[i]);
      careful = __syncthreads_or(odd);
    }
    // ---- O += P V ----
    if (!careful) {
#pragma unroll 4
      for (int j = 0; j < BN; j += 2) {
        float2 p[RM];
#pragma unroll
        for (int i = 0; i < RM; ++i) p[i] = *reinterpret_cast<const float2*>(sp + (ty + 16 * i) * PS + j);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          f32x2 vv[OC / 2];
#pragma unroll
          for (int c = 0; c < OC / 4; ++c) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(sv + (j + u) * D + c * 32 + tx * 4);
            vv[2 * c] = t.x;
            vv[2 * c + 1] = t.y;
          }
#pragma unroll
          for (int i = 0; i < RM; ++i) {
            const float w = u ? p[i].y : p[i].x;
            const f32x2 w2 = pack2(w, w);
#pragma unroll
            for (int c = 0; c < OC / 2; ++c) o[i][c] = fma2(w2, vv[c], o[i][c]);
          }
        }
      }
    } else {
      for (int j = 0; j < BN; ++j)
#pragma unroll
        for (int i = 0; i < RM; ++i)
          if (j0 + j < nkeys[i]) {
            const float w = sp[(ty + 16 * i) * PS + j];
            const f32x2 w2 = pack2(w, w);
#pragma unroll
            for (int c = 0; c < OC / 4; ++c) {
              const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(sv + j * D + c * 32 + tx * 4);
              o[i][2 * c] = fma2(w2, t.x, o[i][2 * c]);
              o[i][2 * c + 1] = fma2(w2, t.y, o[i][2 * c + 1]);
            }
          }
    }
    __syncthreads();
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    float sum = l[i];
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const int r = ty + 16 * i;
    if (r >= live) continue;
    const int64_t row = row0 + r;
    const int head = kvh * G + static_cast<int>(row % G);
    if (a.sink != nullptr && nkeys[i] > 0) sum += exp2f(a.sink[head] * 1.4426950408889634f - m[i]);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    float* op = a.out + ((q0 + row / G) * a.Hq + head) * D + tx * 4;
#pragma unroll
    for (int c = 0; c < OC / 4; ++c) {
      const float2 lo = unpack2(o[i][2 * c]), hi = unpack2(o[i][2 * c + 1]);
      *reinterpret_cast<float4*>(op + c * 32) = make_float4(lo.x * inv, lo.y * inv, hi.x * inv, hi.y * inv);
    }
  }
}

template <int D, int RM>
int launch_tiles(const PrefillF32Args& a, int max_seqlen_q, cudaStream_t s) {
  static bool configured[64] = {false};       // racing threads set the same attribute
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(prefill_f32_kernel<D, RM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem_bytes(D, RM))) != cudaSuccess)
      return B200_ERR_LAUNCH;
    configured[dev] = true;
  }
  const int64_t tiles = (static_cast<int64_t>(max_seqlen_q) * (a.Hq / a.Hkv) + RM * 16 - 1) / (RM * 16);
  const int64_t ctas = tiles * a.Hkv * a.num_seqs;
  if (ctas > 2147483647LL) return B200_ERR_UNSUPPORTED;
  prefill_f32_kernel<D, RM><<<static_cast<unsigned>(ctas), kThreads, smem_bytes(D, RM), s>>>(a);
  return launch_result();
}

template <int D>
int launch_rows(const PrefillF32Args& a, int max_seqlen_q, int64_t total_q, cudaStream_t s) {
  int sms = sm_count_cached();
  if (sms <= 0) sms = 148;
  // tiles of 64 rows move fewer operands per product, tiles of 32 give a small batch more CTAs: the line is where the former
  // still give every SM two (4 prompts of 100 tokens at 16/4 x 64: 18.6 us in tiles of 64, 16.5 us in tiles of 32; 8 prompts
  // of 500 tokens at 16/4 x 32: 79 and 99 us).  Sequences of up to 32 rows fill no more than the smaller tile (256 x 8 tokens behind 64 at
  // 16/16 x 128: 532 us in tiles of 64, 304 in tiles of 32).
  if (static_cast<int64_t>(max_seqlen_q) * (a.Hq / a.Hkv) > 32 && total_q * a.Hq / 64 >= 2 * sms) return launch_tiles<D, 4>(a, max_seqlen_q, s);
  return launch_tiles<D, 2>(a, max_seqlen_q, s);
}

// Whether the general kernel, a warp per row that reads every key, is the faster one: short portions leave most of a 32-row tile
// empty, and a tile of keys costs a CTA as much for one key as for all.  Times of both in us from what they measured at 16/4 x 64, 32/8 x
// 128, 16/16 x 32, 16/16 x 128 and 8/1 x 128, 1 to 256 sequences of 1 to 16 tokens behind 0 to 1,024: a chain of keys or tiles where
// the batch is small, the rate of all warps or CTAs where it is large.  64 x 1 token at 16/4 x 64: 3.2 us, in tiles 10.6; 256 x 1 behind 64 at
// 16/16 x 128: 172 and 302; 256 x 1 behind 64 at 16/4 x 64: 100 and 61.
bool general_is_faster(const PrefillF32Args& a, int D, int64_t total_q, int max_seqlen_q, int max_seqlen_k) {
  const int64_t rows = static_cast<int64_t>(max_seqlen_q) * (a.Hq / a.Hkv);
  if (rows > 32 || max_seqlen_k > 128 || a.num_seqs > 65535 || a.Hq > 65535) return false;      // the latter two: its grid
  const double rate = max_seqlen_q == 1 ? 1600 : max_seqlen_q <= 3 ? 2100 : 3100;                   // rows x keys a us
  const double all = static_cast<double>(total_q) * a.Hq * (max_seqlen_k - max_seqlen_q / 2) / rate;
  const double chain = 0.75 * max_seqlen_k, general = 2.5 + (all > chain ? all : chain);
  const int tiles = (max_seqlen_k + tile_keys(D) - 1) / tile_keys(D);
  const double tile_all = static_cast<double>(a.num_seqs) * a.Hkv * (tiles + 0.5) / (D == 128 ? 41 : D == 64 ? 38 : 75);
  const double tile_chain = 3 + (D == 32 ? 4.2 : 7.5) * tiles;
  return general < 0.9 * (tile_all > tile_chain ? tile_all : tile_chain);
}

}  // namespace

// B200_ERR_UNSUPPORTED: a shape, stride or alignment that the tiles do not take, or sizes at which the general kernel is the faster one
int prefill_f32_launch(const void* q, const void* k, const void* v, void* out, int64_t q_stride, int64_t k_stride,
                       int64_t v_stride, int64_t total_q, const int32_t* cu_q, const int32_t* cu_k, int num_seqs,
                       int max_seqlen_q, int max_seqlen_k, int Hq, int Hkv, int Dqk, int Dv, float scale, const void* kc,
                       const void* vc, const int32_t* bt, int64_t bt_stride, int bs, int64_t num_blocks, const float* sink, int32_t* status,
                       cudaStream_t s) {
  if (Dqk != Dv || (Dqk != 32 && Dqk != 64 && Dqk != 128) || static_cast<int64_t>(num_seqs) * Hkv > 2147483647LL) return B200_ERR_UNSUPPORTED;
  const void* kp = bt ? kc : k;
  const void* vp = bt ? vc : v;
  if (!aligned16(q) || !aligned16(kp) || !aligned16(vp) || !aligned16(out) || q_stride % 4 ||
      (!bt && (k_stride % 4 || v_stride % 4)))
    return B200_ERR_UNSUPPORTED;
  PrefillF32Args a{static_cast<const float*>(q), static_cast<const float*>(kp), static_cast<const float*>(vp),
                   static_cast<float*>(out), q_stride, k_stride, v_stride, cu_q, cu_k, num_seqs, Hq, Hkv,
                   scale * 1.4426950408889634f, bt, bt_stride, bs, num_blocks, sink, status};
  if (general_is_faster(a, Dqk, total_q, max_seqlen_q, max_seqlen_k)) return B200_ERR_UNSUPPORTED;
  if (Dqk == 32) return launch_rows<32>(a, max_seqlen_q, total_q, s);
  if (Dqk == 64) return launch_rows<64>(a, max_seqlen_q, total_q, s);
  return launch_rows<128>(a, max_seqlen_q, total_q, s);
}

}  // namespace b200
