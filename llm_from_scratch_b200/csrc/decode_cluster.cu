// Paged GQA decode attention in bf16, head size 128, for batches that a streaming launch does not fill (paged_decode.cu has the other form and the
// rule): a cluster of CTAs per (sequence, KV head).
//
// The flat cut of paged_decode.cu streams at the rate of the memory, but a small batch spends its time around that: every CTA
// sums all context lengths to find its range, partial results go through global memory, and a second kernel or a counter
// merges them.  Here a CTA knows its share from its own context alone, a warp takes every fourth 16-token block of it, and
// the pieces meet in shared memory, then in the cluster's distributed shared memory.  What is left is one chain of
// latencies: length, block numbers, rows, products, barrier.
//
// Products and softmax are those of the other kernel: the G query heads are the N dimension of mma.sync m16n8k16, S^T = K Q^T and
// O^T = V^T P^T, scores and sums in fp32.  The rows of a block arrive by cp.async, swizzled, two blocks ahead.  Without scratch in global memory
// concurrent calls share nothing.
#include <cooperative_groups.h>

#include "common.cuh"

namespace b200 {
namespace {

namespace cg = cooperative_groups;

struct ClusterArgs {
  const __nv_bfloat16* q;
  const uint8_t* kc;
  const uint8_t* vc;
  __nv_bfloat16* out;
  const int32_t* bt;
  int64_t bt_stride;
  const int64_t* lens;
  int Hq, Hkv, sub;          // sub: 16-token blocks per block-table entry
  int64_t num_blocks;
  float scale_log2;
  const float* sink;         // [Hq] or null
  int32_t* status;
};

constexpr int kDim = 128, kWarps = 4, kThreads = kWarps * 32, kTok = 16;

template <int NT>
struct ClusterLayout {
  static constexpr int D = kDim;
  static constexpr int tile = kTok * D * 2;                           // K or V rows of a block
  static constexpr int stages = 3;                                    // blocks of a warp in flight; two CTAs fit an SM
  static constexpr int ring = kWarps * stages * 2 * tile;
  static constexpr int LDO = D + 4;
  static constexpr int pieces = kWarps * NT * 8 * LDO * 4;            // over the ring
  static constexpr int bytes = ring > pieces ? ring : pieces;
};

template <int NT>
__global__ void __launch_bounds__(kThreads) decode_cluster_kernel(const ClusterArgs a) {
  using L = ClusterLayout<NT>;
  constexpr int D = kDim, ROWB = D * 2, CPR = D / 8, KS = D / 16, LOADS = kTok * CPR / 32, kStages = L::stages;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float s_m[kWarps][NT * 8], s_l[kWarps][NT * 8];
  __shared__ __align__(16) float c_o[NT * 8][D];       // of the CTA, read by the cluster
  __shared__ float c_m[NT * 8], c_l[NT * 8];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = cluster.block_rank(), ranks = cluster.num_blocks();
  const int seq = blockIdx.z, h = blockIdx.y, G = a.Hq / a.Hkv;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  auto swizzle = [](int c, int t) { return c ^ (t & 7); };

  uint32_t qf[NT][KS][2];                              // in flight with the length
  const __nv_bfloat16* qp = a.q + (static_cast<int64_t>(seq) * a.Hq + h * G) * D;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const int head = nt * 8 + g;
      const uint32_t* src = reinterpret_cast<const uint32_t*>(qp + head * D + ks * 16 + tq * 2);
      qf[nt][ks][0] = head < G ? __ldg(src) : 0u;
      qf[nt][ks][1] = head < G ? __ldg(src + 4) : 0u;
    }
  int64_t len64 = a.lens[seq];
  const int64_t cap = a.bt_stride * a.sub * kTok;
  if (len64 > cap) {
    if (tid == 0) report(a.status, B200_ERR_BOUNDS);   // table row too short for the context
    len64 = cap;
  }
  const int len = len64 > 0 ? static_cast<int>(len64) : 0;
  // ---- this CTA's blocks, of them every kWarps-th for a warp.  The first `used` CTAs share the context, a block per warp at least;
  // the others leave: a barrier of the cluster counts the threads that are still there, and nobody reads what they hold.
  const int blocks = (len + kTok - 1) / kTok, per = max((blocks + ranks - 1) / ranks, kWarps), used = max((blocks + per - 1) / per, 1);
  if (rank >= used) return;
  const int lo = min(rank * per, blocks) + warp, hi = min((rank + 1) * per, blocks);
  const int mine = lo < hi ? (hi - lo + kWarps - 1) / kWarps : 0;
  const int32_t* table = a.bt + static_cast<int64_t>(seq) * a.bt_stride;
  const uint32_t ring = smem_u32(smem) + warp * (kStages * 2 * L::tile);
  const int64_t row_stride = static_cast<int64_t>(a.Hkv) * ROWB;
  const uint8_t* kbase = a.kc + static_cast<int64_t>(h) * ROWB;
  const uint8_t* vbase = a.vc + static_cast<int64_t>(h) * ROWB;
  int id_lane = -1;                                    // block number of this lane's block of the current 32
  auto issue = [&](int i) {
    if (i % 32 == 0) {
      const int blk = lo + (i + lane) * kWarps;
      id_lane = -1;
      if (blk < hi) {
        id_lane = __ldg(table + (a.sub == 1 ? blk : blk / a.sub));
        if (static_cast<uint64_t>(static_cast<int64_t>(id_lane)) >= static_cast<uint64_t>(a.num_blocks)) {
          report(a.status, B200_ERR_BOUNDS);
          id_lane = -1;
        }
      }
    }
    const int id = __shfl_sync(0xffffffffu, id_lane, i % 32), blk = lo + i * kWarps;
    const int valid = id >= 0 ? len - blk * kTok : 0;  // tokens to read; rows behind them are zeros
    const int64_t at = id >= 0 ? (static_cast<int64_t>(id) * a.sub + (a.sub == 1 ? 0 : blk % a.sub)) * kTok * row_stride : 0;
    const uint32_t kdst = ring + i % kStages * (2 * L::tile), vdst = kdst + L::tile;
#pragma unroll
    for (int j = 0; j < LOADS; ++j) {
      const int idx = lane + 32 * j, t = idx / CPR, c = idx % CPR;
      const int bytes = t < valid ? 16 : 0;
      const int64_t off = at + (bytes ? t * row_stride + c * 16 : 0);
      const uint32_t d = t * ROWB + swizzle(c, t) * 16;
      cp_async16(kdst + d, kbase + off, bytes);
      cp_async16(vdst + d, vbase + off, bytes);
    }
  };
  float o[NT][KS][4], m[NT][2], l[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    m[nt][0] = m[nt][1] = -INFINITY;
    l[nt][0] = l[nt][1] = 0.f;
#pragma unroll
    for (int mt = 0; mt < KS; ++mt) o[nt][mt][0] = o[nt][mt][1] = o[nt][mt][2] = o[nt][mt][3] = 0.f;
  }
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < mine) issue(s);
    cp_async_commit();
  }
  for (int i = 0; i < mine; ++i) {
    if (i + kStages - 1 < mine) issue(i + kStages - 1);
    cp_async_commit();
    cp_async_wait<kStages - 1>();
    __syncwarp();
    const uint32_t kt = ring + i % kStages * (2 * L::tile), vt = kt + L::tile;
    const int valid = len - (lo + i * kWarps) * kTok;
    // ---- S^T[token, head] = K Q^T
    float s[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
    {
      const int t = (lane & 7) + ((lane >> 3) & 1) * 8, ch = lane >> 4;
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t af[4];
        ldmatrix_x4(af, kt + t * ROWB + swizzle(2 * ks + ch, t) * 16);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_bf16_16816(s[nt], af, qf[nt][ks]);
      }
    }
    // ---- online softmax over the tokens g, g + 8
    uint32_t pb[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = g + 8 * (e >> 1) < valid ? s[nt][e] * a.scale_log2 : -INFINITY;
      float mx[2] = {fmaxf(x[0], x[2]), fmaxf(x[1], x[3])};
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) {
        mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], off));
        mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], off));
      }
      float p[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float mn = fmaxf(m[nt][e], mx[e]), ref = mn == -INFINITY ? 0.f : mn;     // scores of -inf alone: weights 0
        const float al = fast_exp2(m[nt][e] - ref);
        m[nt][e] = mn;
        p[e] = fast_exp2(x[e] - ref);
        p[e + 2] = fast_exp2(x[e + 2] - ref);
        l[nt][e] = l[nt][e] * al + p[e] + p[e + 2];
#pragma unroll
        for (int mt = 0; mt < KS; ++mt) {
          o[nt][mt][e] *= al;
          o[nt][mt][e + 2] *= al;
        }
      }
      pb[nt][0] = movmatrix_trans(pack_bf16x2(p[0], p[1]));
      pb[nt][1] = movmatrix_trans(pack_bf16x2(p[2], p[3]));
    }
    // ---- O^T[d, head] += V^T P^T
    {
      const int t = (lane & 7) + (lane >> 4) * 8, ch = (lane >> 3) & 1;
#pragma unroll
      for (int mt = 0; mt < KS; ++mt) {
        uint32_t af[4];
        ldmatrix_x4_trans(af, vt + t * ROWB + swizzle(2 * mt + ch, t) * 16);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_bf16_16816(o[nt][mt], af, pb[nt]);
      }
    }
    __syncwarp();                                      // the stage may be refilled
  }
  cp_async_wait<0>();
  __syncthreads();                                     // the ring becomes the warps' pieces
  // ---- warps of the CTA
  float* pieces = reinterpret_cast<float*>(smem);
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int head = nt * 8 + tq * 2 + e;
      float sum = l[nt][e];
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
      float* row = pieces + (warp * NT * 8 + head) * L::LDO + g;
#pragma unroll
      for (int mt = 0; mt < KS; ++mt) {
        row[mt * 16] = o[nt][mt][e];
        row[mt * 16 + 8] = o[nt][mt][e + 2];
      }
      if (g == 0) s_m[warp][head] = m[nt][e], s_l[warp][head] = sum;
    }
  __syncthreads();
  for (int i = tid; i < G * (D / 4); i += kThreads) {
    const int head = i / (D / 4), d = i % (D / 4) * 4;
    float M = s_m[0][head];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, s_m[w][head]);
    float sum = 0.f;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = s_m[w][head] == -INFINITY ? 0.f : exp2f(s_m[w][head] - M);
      const float4 y = *reinterpret_cast<const float4*>(pieces + (w * NT * 8 + head) * L::LDO + d);
      x.x += f * y.x, x.y += f * y.y, x.z += f * y.z, x.w += f * y.w;
      sum += f * s_l[w][head];
    }
    *reinterpret_cast<float4*>(&c_o[head][d]) = x;
    if (d == 0) c_m[head] = M, c_l[head] = sum;
  }
  if (used > 1) cluster.sync();
  else __syncthreads();
  // ---- CTAs of the cluster: every one finishes its share of the columns
  for (int i = rank * kThreads + tid; i < G * (D / 2); i += used * kThreads) {
    const int head = i / (D / 2), d = i % (D / 2) * 2;
    float mr[8], lr[8], M = -INFINITY;
    float2 y[8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < used) {
        mr[r] = *cluster.map_shared_rank(&c_m[head], r);
        lr[r] = *cluster.map_shared_rank(&c_l[head], r);
        y[r] = *reinterpret_cast<const float2*>(cluster.map_shared_rank(&c_o[head][d], r));
        M = fmaxf(M, mr[r]);
      }
    float sum = 0.f, x0 = 0.f, x1 = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < used) {
        const float f = mr[r] == -INFINITY ? 0.f : exp2f(mr[r] - M);
        sum += f * lr[r];
        x0 += f * y[r].x;
        x1 += f * y[r].y;
      }
    if (a.sink != nullptr && M > -INFINITY) sum += sink_term(a.sink[h * G + head], M);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;     // an empty context gives zeros
    *reinterpret_cast<uint32_t*>(a.out + (static_cast<int64_t>(seq) * a.Hq + h * G + head) * D + d) = pack_bf16x2(x0 * inv, x1 * inv);
  }
  if (used > 1) cluster.sync();                        // nobody leaves while another CTA reads its shared memory
}

template <int NT>
int launch(const ClusterArgs& a, int batch, int ranks, cudaStream_t s) {
  constexpr int smem = ClusterLayout<NT>::bytes;
  static bool configured[64] = {false};                // racing threads set the same attribute
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(decode_cluster_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return B200_ERR_LAUNCH;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ranks, a.Hkv, batch);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return launch_result(cudaLaunchKernelEx(&cfg, decode_cluster_kernel<NT>, a));
}

}  // namespace

// For the shapes of the fast plan of paged_decode.cu.  B200_ERR_UNSUPPORTED: the streaming form takes them.
int decode_cluster_launch(const void* q, const void* kc, const void* vc, void* out, const int32_t* bt, int64_t bt_stride,
                          const int64_t* lens, int batch, int Hq, int Hkv, int D, int sub, int64_t num_blocks, float scale_log2,
                          const float* sink, int32_t* status, cudaStream_t s) {
  const int sms = sm_count_cached();
  // Head size 128.  At 64 a call is as much faster (64 x 64 .. 1,024 tokens at 16/4 heads: 13 against 19 us), but its bf16 weights
  // round at other places, and behind the 16 expert layers of the decoder that has heads of 64 that moves logits by 4 %.
  if (D != kDim || sms <= 0 || batch > 65535) return B200_ERR_UNSUPPORTED;
  const int64_t pairs = static_cast<int64_t>(batch) * Hkv, keys = bt_stride * sub * kTok, wave = 2 * static_cast<int64_t>(sms);
  // CTAs per context: one wave of them, none with less than a block per warp; where a context may leave a CTA more than 1,024
  // tokens up to two waves, which evens out unequal contexts (16 of 128 .. 8,192 tokens: four CTAs 36 us, two 48, one 76; with
  // four waves 32 short contexts under a wide table took longer than in one stream: 256 tokens 18 against 14 us).
  int ranks = 1;
  while (ranks < 8 && static_cast<int64_t>(ranks) * kWarps * kTok < keys && pairs * ranks * 2 <= wave * (keys / ranks > 1024 ? 2 : 1))
    ranks *= 2;
  // Only the width of the table is known here, so the line lies where no contexts that fit it are slower than in one stream by more
  // than the stream's own scatter.  Times in us, clusters / stream, 32/8 heads; `64+n`: one context of n tokens among those of 64.
  //   one context of 700 tokens 5.5 / 16, of 8,192 13 / 70; 16 of 64 4.1 / 7.8, of 2,000 23 / 37
  //   32 (256 pairs): of 64 4.6 / 8.0, of 700 12.4 / 24; under a table of 8,192 (two CTAs each) of 128 .. 8,192 72 / 70
  //   64 (512 pairs): of 64 7.6 / 9.0, of 64 .. 1,024 21 / 24, but 64+4000 41 / 25
  //   128 (1,024 pairs): of 64 13.5 / 9.2, of 700 62 / 65; 512: of 16 41 / 14, of 700 215 / 228
  if (keys > (pairs * 2 <= wave ? 32768 : pairs <= wave ? 8192 : pairs <= 2 * wave ? 2048 : 0)) return B200_ERR_UNSUPPORTED;
  const ClusterArgs a{static_cast<const __nv_bfloat16*>(q), static_cast<const uint8_t*>(kc), static_cast<const uint8_t*>(vc),
                      static_cast<__nv_bfloat16*>(out), bt, bt_stride, lens, Hq, Hkv, sub, num_blocks, scale_log2, sink, status};
  return Hq / Hkv > 8 ? launch<2>(a, batch, ranks, s) : launch<1>(a, batch, ranks, s);
}

}  // namespace b200
