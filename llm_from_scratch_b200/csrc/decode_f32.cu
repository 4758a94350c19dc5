// Paged GQA decode attention in fp32: head sizes 32, 64 and 128, any page size, optional sinks.
//
// Bound by reading every K and V row of every context once.  A CTA takes up to four query heads of one KV head, so a row serves
// all of them, and a cluster of CTAs shares the context of a sequence, whose partial results meet through distributed shared
// memory.  There is no scratch in global memory, so calls on different streams have nothing in common.  D / 8 lanes hold
// a token: eight channels of its K and V row and of every head's query and output each.  The sums of a trip's (token, head)
// pairs over those lanes are transposed on the way, so that a lane ends with one to four scores and takes their exponentials.
// A lane copies its own pieces of the rows a trip ahead into a ring of its own; the block numbers of a CTA's range are
// read into shared memory first, because a table read per trip, even one trip ahead, set the pace.
//
// Measured at 64 sequences of 64 to 1024 tokens, 16/4 heads x 64: 28 us (the general kernel, a CTA per sequence and query
// head: 307 us); 128 sequences of 2048 tokens, 32/8 x 128: 346 us, 6.2 TB/s.  With the table read inside the trips and a full
// reduction of every score the latter took 457 us.
#include <cooperative_groups.h>

#include "sequences.cuh"

namespace b200 {
namespace {

namespace cg = cooperative_groups;

struct DecodeF32Args {
  const float* q;
  const float* kc;
  const float* vc;
  float* out;
  const int32_t* bt;
  int64_t bt_stride;
  const int64_t* lens;
  int Hq, Hkv, bs;
  int64_t num_blocks;
  float scale_log2;
  const float* sink;         // [Hq] or null
  int32_t* status;
};

constexpr int kWarps = 4, kThreads = kWarps * 32;
constexpr int kUnroll = 4;   // tokens of a lane group per trip: 8 KB of a warp
constexpr int kStages = 2;   // trips in flight
constexpr int kTable = 1024; // block numbers held at a time
constexpr size_t kRingBytes = static_cast<size_t>(kWarps) * kStages * kUnroll * 4 * 32 * sizeof(float4);

// GC: query heads of the CTA
template <int D, int GC>
__global__ void __launch_bounds__(kThreads, 3) decode_f32_kernel(const DecodeF32Args a) {
  constexpr int LP = D / 8;                    // lanes of a token
  constexpr int TW = 32 / LP;                  // tokens of a warp
  extern __shared__ float4 ring[];             // [warp][stage][token, K | V, half][lane]
  __shared__ __align__(16) float s_o[kWarps][GC][D];
  __shared__ float s_m[kWarps][GC], s_l[kWarps][GC];
  __shared__ __align__(16) float c_o[GC][D];   // of the CTA, read by the cluster's first one
  __shared__ float c_m[GC], c_l[GC];
  __shared__ int s_table[kTable];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = cluster.block_rank(), ranks = cluster.num_blocks();
  const int seq = blockIdx.z, head0 = blockIdx.y * GC, kvh = head0 / (a.Hq / a.Hkv);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sub = lane % LP, grp = lane / LP;
  int64_t len64 = a.lens[seq];
  const int64_t cap = a.bt_stride * a.bs;
  if (len64 > cap) {
    if (tid == 0) report(a.status, B200_ERR_BOUNDS);
    len64 = cap;
  }
  const int len = len64 > 0 ? static_cast<int>(len64) : 0;
  const int32_t* table = a.bt + static_cast<int64_t>(seq) * a.bt_stride;

  // lane `sub` of a token ends up with the scores of the pairs own, own + 1, ... of a trip
  constexpr int NV = kUnroll * GC, OWN = NV > LP ? NV / LP : 1;
  const int own = sub * NV / LP;
  f32x2 q[GC][4], o[GC][4];                    // channels 4 sub .. and 4 (sub + LP) ..
  float m[GC], m_own[OWN], l_own[OWN];
#pragma unroll
  for (int g = 0; g < GC; ++g) {
    const float4* qp = reinterpret_cast<const float4*>(a.q + (static_cast<int64_t>(seq) * a.Hq + head0 + g) * D);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float4 x = qp[sub + c * LP];
      q[g][2 * c] = pack2(x.x * a.scale_log2, x.y * a.scale_log2);
      q[g][2 * c + 1] = pack2(x.z * a.scale_log2, x.w * a.scale_log2);
      o[g][2 * c] = o[g][2 * c + 1] = 0;
    }
    m[g] = -INFINITY;
  }
#pragma unroll
  for (int c = 0; c < OWN; ++c) m_own[c] = -INFINITY, l_own[c] = 0.f;

  // ---- the CTA's range of the context
  constexpr int TRIP = kWarps * TW * kUnroll;
  const int per = ((len + ranks - 1) / ranks + TRIP - 1) / TRIP * TRIP;
  const int used = per > 0 ? (len + per - 1) / per : 1;       // CTAs with keys; a barrier of the cluster does not count those that left
  if (rank >= used) return;
  const int lo = min(rank * per, len), hi = min(lo + per, len);
  const int shift = (a.bs & (a.bs - 1)) == 0 ? __ffs(a.bs) - 1 : -1;
  auto page_of = [&](int t) { return shift >= 0 ? t >> shift : t / a.bs; };
  float4* slots = ring + (warp * kStages * kUnroll * 4) * 32 + lane;
  const int span = static_cast<int>(min(static_cast<int64_t>(kTable - 1) * a.bs, static_cast<int64_t>(len)));
  for (int base = lo; base < hi; base += span) {
    const int end = min(base + span, hi), page0 = page_of(base), pages = page_of(end - 1) - page0 + 1;
    __syncthreads();
    for (int i = tid; i < pages; i += kThreads) {
      int id = table[page0 + i];
      if (static_cast<uint64_t>(static_cast<int64_t>(id)) >= static_cast<uint64_t>(a.num_blocks)) {
        report(a.status, B200_ERR_BOUNDS);
        id = -1;
      }
      s_table[i] = id;
    }
    __syncthreads();
    const int first = base + warp * kUnroll * TW + grp;     // token u of this lane group's trip i: first + i * TRIP + u * TW
    const int trips = (end - (base + warp * kUnroll * TW) + TRIP - 1) / TRIP;        // the same for all lanes of the warp
    uint32_t valid = 0;                          // of the tokens in flight, kUnroll bits a trip, the latest trip in the low ones
    auto issue = [&](int i) {
      float4* dst = slots + (i % kStages) * kUnroll * 4 * 32;
      valid <<= kUnroll;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int t = first + i * TRIP + u * TW, page = page_of(min(t, end - 1)), id = s_table[page - page0];
        const bool in = t < end && id >= 0;
        if (in) valid |= 1u << u;
        const int64_t row = in ? ((static_cast<int64_t>(id) * a.bs + (t - page * a.bs)) * a.Hkv + kvh) * D + sub * 4 : 0;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          cp_async16(smem_u32(dst + (u * 4 + c) * 32), a.kc + row + (in ? c * LP * 4 : 0), in ? 16 : 0);
          cp_async16(smem_u32(dst + (u * 4 + 2 + c) * 32), a.vc + row + (in ? c * LP * 4 : 0), in ? 16 : 0);
        }
      }
    };
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) {
      if (i < trips) issue(i);
      else valid <<= kUnroll;
      cp_async_commit();
    }
    for (int i = 0; i < trips; ++i) {
      if (i + kStages - 1 < trips) issue(i + kStages - 1);
      else valid <<= kUnroll;
      cp_async_commit();
      cp_async_wait<kStages - 1>();              // a lane reads only what it copied itself
      const float4* src = slots + (i % kStages) * kUnroll * 4 * 32;
      const uint32_t bits = valid >> ((kStages - 1) * kUnroll);
      // ---- scores: pair v = u * GC + g
      float x[NV];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        f32x2 k[4];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + (u * 4 + c) * 32);
          k[2 * c] = t.x, k[2 * c + 1] = t.y;
        }
#pragma unroll
        for (int g = 0; g < GC; ++g) {
          f32x2 acc = mul2(q[g][0], k[0]);
#pragma unroll
          for (int c = 1; c < 4; ++c) acc = fma2(q[g][c], k[c], acc);
          const float2 h = unpack2(acc);
          x[u * GC + g] = h.x + h.y;
        }
      }
      // sums over the LP lanes; every step a lane keeps half of the pairs it still has
      {
        int n = NV;
#pragma unroll
        for (int off = LP / 2; off >= 1; off >>= 1) {
          if (n > 1) {
            n /= 2;
            const bool up = sub & off;
#pragma unroll
            for (int c = 0; c < NV / 2; ++c)
              if (c < n) {
                const float send = up ? x[c] : x[c + n], keep = up ? x[c + n] : x[c];
                x[c] = keep + __shfl_xor_sync(0xffffffffu, send, off);
              }
          } else {
            x[0] += __shfl_xor_sync(0xffffffffu, x[0], off);
          }
        }
      }
      bool in[OWN], grows = false;
#pragma unroll
      for (int c = 0; c < OWN; ++c) {
        in[c] = bits >> ((own + c) / GC) & 1;
        if (!in[c]) x[c] = -INFINITY;
        grows |= in[c] && !(x[c] <= m_own[c]);
      }
      if (__any_sync(0xffffffffu, grows)) {
        float al_own[OWN];
#pragma unroll
        for (int g = 0; g < GC; ++g) {
          float mn = m[g];
#pragma unroll
          for (int u = 0; u < kUnroll; ++u)
            mn = fmaxf(mn, __shfl_sync(0xffffffffu, x[(u * GC + g) % OWN], (u * GC + g) * LP / NV, LP));
          const float al = mn == m[g] ? 1.f : fast_exp2(m[g] - mn);
          m[g] = mn;
          const f32x2 al2 = pack2(al, al);
#pragma unroll
          for (int c = 0; c < 4; ++c) o[g][c] = mul2(o[g][c], al2);
#pragma unroll
          for (int c = 0; c < OWN; ++c)
            if ((own + c) % GC == g) m_own[c] = mn, al_own[c] = al;
        }
#pragma unroll
        for (int c = 0; c < OWN; ++c) l_own[c] *= al_own[c];
      }
      float p[OWN];
#pragma unroll
      for (int c = 0; c < OWN; ++c) {
        p[c] = x[c] == -INFINITY ? 0.f : fast_exp2(x[c] - m_own[c]);       // a maximum of -inf must not meet another
        l_own[c] += p[c];
      }
      // ---- outputs
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        f32x2 v[4];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + (u * 4 + 2 + c) * 32);
          v[2 * c] = t.x, v[2 * c + 1] = t.y;
        }
#pragma unroll
        for (int g = 0; g < GC; ++g) {
          const float w = __shfl_sync(0xffffffffu, p[(u * GC + g) % OWN], (u * GC + g) * LP / NV, LP);
          const f32x2 w2 = pack2(w, w);
#pragma unroll
          for (int c = 0; c < 4; ++c) o[g][c] = fma2(w2, v[c], o[g][c]);
        }
      }
    }
    cp_async_wait<0>();
  }
  // ---- lane groups of the warp, warps of the CTA, CTAs of the cluster ----
#pragma unroll
  for (int g = 0; g < GC; ++g) {
    float M = m[g];
#pragma unroll
    for (int off = LP; off < 32; off <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    const float w = m[g] == -INFINITY ? 0.f : exp2f(m[g] - M);
    float sum = 0.f;                           // pairs that several lanes hold count once
#pragma unroll
    for (int c = 0; c < OWN; ++c)
      if ((own + c) % GC == g && (NV >= LP || sub % (LP / NV ? LP / NV : 1) == 0)) sum += l_own[c] * w;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 lo2 = unpack2(o[g][2 * c]), hi2 = unpack2(o[g][2 * c + 1]);
      float4 x = make_float4(lo2.x * w, lo2.y * w, hi2.x * w, hi2.y * w);
#pragma unroll
      for (int off = LP; off < 32; off <<= 1) {
        x.x += __shfl_xor_sync(0xffffffffu, x.x, off);
        x.y += __shfl_xor_sync(0xffffffffu, x.y, off);
        x.z += __shfl_xor_sync(0xffffffffu, x.z, off);
        x.w += __shfl_xor_sync(0xffffffffu, x.w, off);
      }
      if (grp == 0) *reinterpret_cast<float4*>(&s_o[warp][g][(sub + c * LP) * 4]) = x;
    }
    if (lane == 0) s_m[warp][g] = M, s_l[warp][g] = sum;
  }
  __syncthreads();
  for (int i = tid; i < GC * D; i += kThreads) {
    const int g = i / D, d = i % D;
    float M = s_m[0][g];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, s_m[w][g]);
    float x = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = s_m[w][g] == -INFINITY ? 0.f : exp2f(s_m[w][g] - M);
      x += f * s_o[w][g][d];
      sum += f * s_l[w][g];
    }
    c_o[g][d] = x;
    if (d == 0) c_m[g] = M, c_l[g] = sum;
  }
  if (used > 1) cluster.sync();
  else __syncthreads();
  // every CTA finishes its share of the columns
  for (int i = rank * kThreads + tid; i < GC * D; i += used * kThreads) {
    const int g = i / D, d = i % D;
    float M = -INFINITY;
    for (int r = 0; r < used; ++r) M = fmaxf(M, *cluster.map_shared_rank(&c_m[g], r));
    float x = 0.f, sum = 0.f;
    for (int r = 0; r < used; ++r) {
      const float mr = *cluster.map_shared_rank(&c_m[g], r);
      const float f = mr == -INFINITY ? 0.f : exp2f(mr - M);
      x += f * *cluster.map_shared_rank(&c_o[g][d], r);
      sum += f * *cluster.map_shared_rank(&c_l[g], r);
    }
    if (a.sink != nullptr && M > -INFINITY) sum += exp2f(a.sink[head0 + g] * 1.4426950408889634f - M);
    a.out[(static_cast<int64_t>(seq) * a.Hq + head0 + g) * D + d] = sum == 0.f ? 0.f : x / sum;   // 0: no key; a NaN stays one
  }
  if (used > 1) cluster.sync();            // nobody leaves while another CTA reads its shared memory
}

template <int D, int GC>
int launch_heads(const DecodeF32Args& a, int batch, int ranks, cudaStream_t s) {
  static bool configured[64] = {false};       // racing threads set the same attribute
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(decode_f32_kernel<D, GC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kRingBytes)) != cudaSuccess)
      return B200_ERR_LAUNCH;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ranks, a.Hq / GC, batch);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kRingBytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return launch_result(cudaLaunchKernelEx(&cfg, decode_f32_kernel<D, GC>, a));
}

template <int D>
int launch_dim(const DecodeF32Args& a, int batch, cudaStream_t s) {
  int sms = sm_count_cached();
  if (sms <= 0) sms = 148;
  const int G = a.Hq / a.Hkv, GC = G % 4 == 0 ? 4 : G % 2 == 0 ? 2 : 1;
  // CTAs per context: doubled up to four an SM, none with less than a trip of its own; where contexts may be long, up to eight an SM,
  // which evens out batches of unequal contexts.  Three CTAs fit an SM at head sizes 32 and 64, two at 128, so four are more than one
  // round; the line is where the times lie, not a wave (one, two, four, eight CTAs per context, 64 .. 1,024 tokens: 64 sequences at 16/4 x
  // 64 19.5, 17.0, 19.2, 25.8 us, 32 at 32/8 x 128 34, 32, 38, 52; 128 .. 8,192 tokens, 64 at 16/4 x 64 129, 75, 64, 65).
  const int64_t pairs = static_cast<int64_t>(batch) * (a.Hq / GC), keys = a.bt_stride * a.bs;
  // The general kernel keeps contexts of up to eight tokens, where the merges are the call (one token at 16/4 x 64: 4.7 against 2.8 us), and
  // large batches of up to sixteen where no heads share the rows (256 x 16 at 16/16 x 32: 28 against 19).
  if (keys <= 8 || (keys <= 16 && GC == 1 && pairs >= 2048)) return B200_ERR_UNSUPPORTED;
  const int trip = kWarps * (32 / (D / 8)) * kUnroll;
  int ranks = 1;
  while (ranks < 8 && static_cast<int64_t>(ranks) * trip < keys &&
         pairs * ranks * 2 <= (keys / ranks > 1024 ? 8 : 4) * static_cast<int64_t>(sms))
    ranks *= 2;
  if (GC == 4) return launch_heads<D, 4>(a, batch, ranks, s);
  if (GC == 2) return launch_heads<D, 2>(a, batch, ranks, s);
  return launch_heads<D, 1>(a, batch, ranks, s);
}

}  // namespace

// B200_ERR_UNSUPPORTED: a shape or alignment that the general kernel takes, or contexts too short for clusters
int decode_f32_launch(const void* q, const void* kc, const void* vc, void* out, const int32_t* bt, int64_t bt_stride,
                      const int64_t* lens, int batch, int Hq, int Hkv, int D, int Dv, int bs, int64_t num_blocks,
                      float scale_log2, const float* sink, int32_t* status, cudaStream_t s) {
  if (D != Dv || (D != 32 && D != 64 && D != 128) || !aligned16(q) || !aligned16(kc) || !aligned16(vc) || !aligned16(out) ||
      batch > 65535 || Hq > 65535)
    return B200_ERR_UNSUPPORTED;
  DecodeF32Args a{static_cast<const float*>(q), static_cast<const float*>(kc), static_cast<const float*>(vc),
                  static_cast<float*>(out), bt, bt_stride, lens, Hq, Hkv, bs, num_blocks, scale_log2, sink, status};
  if (D == 32) return launch_dim<32>(a, batch, s);
  if (D == 64) return launch_dim<64>(a, batch, s);
  return launch_dim<128>(a, batch, s);
}

}  // namespace b200
