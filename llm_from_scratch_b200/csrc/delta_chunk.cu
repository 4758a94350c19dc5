// Gated delta rule of prompts and portions on tensor cores: sequences are cut into chunks of 64 tokens, and within a chunk
// the 64 dependent rank-one updates become one triangular solve.  With b_i the running sum of ln g inside the chunk,
// gamma_i = exp(b_i), S the state at the chunk's start and K, Q, V the chunk's rows (K, Q behind silu, not yet of unit
// length; rk_i, rq_i their reciprocal norms, rq_i with the factor dk^-1/2):
//
//   A_ij = beta_i rk_i rk_j exp(b_i - b_j) (k_i . k_j)   j < i          T = (I + A)^-1 diag(beta)
//   P_ij = rq_i rk_j exp(b_i - b_j) (q_i . k_j)          j <= i
//   U = T (V - diag(gamma rk) K S),   O = diag(gamma rq) Q S + P U,   S' = gamma_C S + K^T diag(rk gamma_C / gamma) U
//
// delta_prepare_kernel  T and P of every (chunk, value head), all in parallel
// delta_scan_kernel, delta_split_kernel
//                       one CTA per (sequence, value head) walks the chunks.  A warp owns 16 value columns of the state for
//                       the whole sequence: S^T [16, dk] stays in registers as accumulators, and because the accumulators
//                       of one product have the layout of the next product's A operand, S^T, U^T and O^T never leave the
//                       registers between the five products.  Norm and output gate follow in the same launch.
//
// Precision: everything behind the activations is fp32.  K, Q and V are bf16 as they come, so they are exact operands, and
// their norms are factors outside the products.  Every fp32 operand (S, U, T, P) is split into three bf16 parts that
// carry 24 bits together: products with one fp32 operand take three tensor-core products, those with two take the six
// that matter; sums are fp32.  Differences of b are taken in double precision.
#include <cuda.h>

#include <type_traits>

#include "delta_common.cuh"
#include "umma.cuh"

namespace b200 {
namespace {

constexpr int C = 64;                          // tokens per chunk
constexpr int kPrepThreads = 128;
// T and P leave their 16 x 16 tiles above the diagonal out; a tile lies in the order of the B operand of mma.sync: the four
// words of a lane side by side, word 2 h + n of lane (g, tq) = elements (g + 8 h, 2 tq + 8 n) and the next
constexpr int kTiles = (C / 16) * (C / 16 + 1) / 2;
constexpr int kPlane = kTiles * 128;           // words of one part of T or P
constexpr int kBlobBytes = 6 * kPlane * 4 + 4 * C * 4;   // T parts, P parts, then four fp32 vectors per token
__host__ __device__ constexpr int tile_of(int r, int c) { return r * (r + 1) / 2 + c; }

struct ChunkArgs {
  DeltaArgs d;
  uint8_t* blobs;                              // [chunks, H] x kBlobBytes
};

// x0, x1 -> three packed bf16 pairs whose sum is x to 24 bits
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16x2(x0, x1);
  x0 -= __uint_as_float(h << 16);
  x1 -= __uint_as_float(h & 0xffff0000u);
  m = pack_bf16x2(x0, x1);
  x0 -= __uint_as_float(m << 16);
  x1 -= __uint_as_float(m & 0xffff0000u);
  l = pack_bf16x2(x0, x1);
}

// A operand of k-step tiles t0, t1 (accumulator layout) in three parts
__device__ __forceinline__ void split_a(const float (&t0)[4], const float (&t1)[4], uint32_t (&h)[4], uint32_t (&m)[4],
                                        uint32_t (&l)[4]) {
  split3(t0[0], t0[1], h[0], m[0], l[0]);
  split3(t0[2], t0[3], h[1], m[1], l[1]);
  split3(t1[0], t1[1], h[2], m[2], l[2]);
  split3(t1[2], t1[3], h[3], m[3], l[3]);
}

template <int DK>
struct PrepSmem {
  static constexpr int ROW = DK + 8;           // padded row, elements
  static constexpr int LDA = C + 4;
  __nv_bfloat16 k[C * ROW], q[C * ROW];
  float a[C * LDA];
  double b[C];
  float rk[C], rq[C], beta[C];
};

template <int DK>
__global__ void __launch_bounds__(kPrepThreads) delta_prepare_kernel(const ChunkArgs args) {
  using Sm = PrepSmem<DK>;
  extern __shared__ __align__(16) uint8_t raw[];
  Sm& sm = *reinterpret_cast<Sm*>(raw);
  const DeltaArgs& a = args.d;
  const int head = blockIdx.y, kh = head / (a.H / a.G), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int seq, index;
  if (!find_segment(a.cu_q, a.n, C, blockIdx.x, &seq, &index)) return;
  SeqInfo info;
  if (!sequence_info(a, seq, &info)) return;
  const int nt = min(C, info.len - index * C);
  const int64_t tok0 = info.tok0 + index * C;
  // ---- K and Q rows, zero beyond the chunk's tokens and beyond dk
  {
    constexpr int CPR = DK / 8;
    const __nv_bfloat16* kp = static_cast<const __nv_bfloat16*>(a.k) + tok0 * a.act_stride + kh * a.dk;
    const __nv_bfloat16* qp = static_cast<const __nv_bfloat16*>(a.q) + tok0 * a.act_stride + kh * a.dk;
    for (int i = tid; i < C * CPR; i += kPrepThreads) {
      const int r = i / CPR, c = i % CPR;
      const bool ok = r < nt && c * 8 < a.dk;
      const int64_t off = ok ? r * a.act_stride + c * 8 : 0;
      cp_async16(smem_u32(sm.k + r * Sm::ROW + c * 8), kp + off, ok ? 16 : 0);
      cp_async16(smem_u32(sm.q + r * Sm::ROW + c * 8), qp + off, ok ? 16 : 0);
    }
    cp_async_commit();
  }
  // ---- running sum of ln g (warp 0, two tokens per lane), write strengths
  if (warp == 0) {
    double g[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = 2 * lane + e;
      float lg = 0.f, beta = 0.f;
      if (t < nt) {
        const int64_t row = (tok0 + t) * a.proj_stride + head;
        lg = log_decay(__bfloat162float(static_cast<const __nv_bfloat16*>(a.a)[row]) + a.dt_bias[head], a.a_log[head]);
        beta = sigmoid_f(__bfloat162float(static_cast<const __nv_bfloat16*>(a.b)[row]));
      }
      g[e] = lg;
      sm.beta[t] = beta;
    }
    double incl = g[0] + g[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    sm.b[2 * lane] = incl - g[1];
    sm.b[2 * lane + 1] = incl;
  }
  cp_async_wait<0>();
  __syncthreads();
  // ---- reciprocal norms: two threads per row
  {
    const int r = tid >> 1;
    float kk = 0.f, qq = 0.f;
    for (int c = (tid & 1) * 8; c < DK; c += 16) {
      const uint4 kv = *reinterpret_cast<const uint4*>(sm.k + r * Sm::ROW + c);
      const uint4 qv = *reinterpret_cast<const uint4*>(sm.q + r * Sm::ROW + c);
      const __nv_bfloat162* k2 = reinterpret_cast<const __nv_bfloat162*>(&kv);
      const __nv_bfloat162* q2 = reinterpret_cast<const __nv_bfloat162*>(&qv);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = __bfloat1622float2(k2[e]), y = __bfloat1622float2(q2[e]);
        kk += x.x * x.x + x.y * x.y;
        qq += y.x * y.x + y.y * y.y;
      }
    }
    kk += __shfl_xor_sync(0xffffffffu, kk, 1);
    qq += __shfl_xor_sync(0xffffffffu, qq, 1);
    if ((tid & 1) == 0) {
      sm.rk[r] = rsqrtf(kk + 1e-6f);
      sm.rq[r] = rsqrtf(qq + 1e-6f) * rsqrtf(static_cast<float>(a.dk));
    }
  }
  __syncthreads();
  uint8_t* blob = args.blobs + (static_cast<size_t>(blockIdx.x) * a.H + head) * kBlobBytes;
  uint32_t* planes = reinterpret_cast<uint32_t*>(blob);
  // ---- K K^T and Q K^T of this warp's 16 rows, columns up to the diagonal
  {
    uint32_t kf[DK / 16][4], qf[DK / 16][4];
    const int r = warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, chalf = lane >> 4;
#pragma unroll
    for (int ks = 0; ks < DK / 16; ++ks) {
      ldmatrix_x4(kf[ks], smem_u32(sm.k + r * Sm::ROW + ks * 16 + chalf * 8));
      ldmatrix_x4(qf[ks], smem_u32(sm.q + r * Sm::ROW + ks * 16 + chalf * 8));
    }
    const int g = lane >> 2, tq = lane & 3, r_in = (lane & 7) + (lane >> 4) * 8, bh = (lane >> 3) & 1;
    for (int p = 0; p <= warp; ++p) {            // 16 columns at a time
      float kk[2][4], qk[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) kk[n][e] = qk[n][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < DK / 16; ++ks) {
        uint32_t bf[4];
        ldmatrix_x4(bf, smem_u32(sm.k + (p * 16 + r_in) * Sm::ROW + ks * 16 + bh * 8));
        const uint32_t b0[2] = {bf[0], bf[1]}, b1[2] = {bf[2], bf[3]};
        mma_bf16_16816(kk[0], kf[ks], b0);
        mma_bf16_16816(kk[1], kf[ks], b1);
        mma_bf16_16816(qk[0], qf[ks], b0);
        mma_bf16_16816(qk[1], qf[ks], b1);
      }
      uint32_t part[3][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = warp * 16 + g + 8 * h, j = p * 16 + n * 8 + 2 * tq;
          float v[2], w[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float dec = j + e <= i ? expf(static_cast<float>(sm.b[i] - sm.b[j + e])) * sm.rk[j + e] : 0.f;
            v[e] = j + e < i ? sm.beta[i] * sm.rk[i] * dec * kk[n][2 * h + e] : 0.f;
            w[e] = sm.rq[i] * dec * qk[n][2 * h + e];
          }
          *reinterpret_cast<float2*>(sm.a + i * Sm::LDA + j) = make_float2(v[0], v[1]);
          split3(w[0], w[1], part[0][2 * h + n], part[1][2 * h + n], part[2][2 * h + n]);
        }
#pragma unroll
      for (int x = 0; x < 3; ++x)
        *reinterpret_cast<uint4*>(planes + (3 + x) * kPlane + tile_of(warp, p) * 128 + lane * 4) =
            make_uint4(part[x][0], part[x][1], part[x][2], part[x][3]);
    }
  }
  __syncthreads();
  // ---- (I + A)^-1, a column per thread by forward substitution; warp 1 starts at row 32
  float* t_rows = reinterpret_cast<float*>(sm.k);      // K and Q are done with
  static_assert(sizeof(sm.k) + sizeof(sm.q) >= C * Sm::LDA * sizeof(float), "T is staged over K and Q");
  if (tid < C) {
    const int j = tid;
    float x[C];
    const float beta = sm.beta[j];
    auto rows = [&](auto lo_c) {
      constexpr int LO = decltype(lo_c)::value;
#pragma unroll
      for (int i = LO; i < C; ++i) {
        float s0 = i == j ? 1.f : 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (int m = LO; m < i; m += 4) {
          const float4 r = *reinterpret_cast<const float4*>(sm.a + i * Sm::LDA + m);   // zero from the diagonal on
          s0 -= r.x * x[m];
          if (m + 1 < i) s1 -= r.y * x[m + 1];
          if (m + 2 < i) s2 -= r.z * x[m + 2];
          if (m + 3 < i) s3 -= r.w * x[m + 3];
        }
        x[i] = (s0 + s1) + (s2 + s3);
      }
#pragma unroll
      for (int i = LO; i < C; ++i) t_rows[i * Sm::LDA + j] = x[i] * beta;
    };
    if (warp == 0) rows(std::integral_constant<int, 0>{});
    else rows(std::integral_constant<int, 32>{});
  } else {
    // ---- factors per token: gamma rq, gamma rk, rk gamma_C / gamma; gamma_C
    const int t = tid - C;
    float* f = reinterpret_cast<float*>(blob + 6 * kPlane * 4);
    const float gamma = expf(static_cast<float>(sm.b[t]));
    f[t] = gamma * sm.rq[t];
    f[C + t] = gamma * sm.rk[t];
    f[2 * C + t] = sm.rk[t] * expf(static_cast<float>(sm.b[C - 1] - sm.b[t]));
    f[3 * C + t] = expf(static_cast<float>(sm.b[C - 1]));
  }
  __syncthreads();
  // ---- T in tiles
  for (int u = tid; u < kTiles * 32; u += kPrepThreads) {
    const int tile = u >> 5, l = u & 31, r = (tile >= 6) + (tile >= 3) + (tile >= 1), c = tile - tile_of(r, 0);
    const float* at = t_rows + (r * 16 + (l >> 2)) * Sm::LDA + c * 16 + 2 * (l & 3);
    uint32_t part[3][4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float2 x = *reinterpret_cast<const float2*>(at + (w >> 1) * 8 * Sm::LDA + (w & 1) * 8);
      split3(x.x, x.y, part[0][w], part[1][w], part[2][w]);
    }
#pragma unroll
    for (int x = 0; x < 3; ++x)
      *reinterpret_cast<uint4*>(planes + x * kPlane + u * 4) = make_uint4(part[x][0], part[x][1], part[x][2], part[x][3]);
  }
}

// Copies of a chunk into shared memory: a thread per row, one for what lies in a piece, counted on an mbarrier.  (16-byte
// cp.async by all threads held up the chain from chunk to chunk for half of its time: 6,600 of 13,000 clocks.)
__device__ __forceinline__ void copy_piece(uint8_t* dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
               "r"(bytes), "r"(bar) : "memory");
}
// For every thread of the CTA, each with whether its wait for the copies counted on `bar` ended: true if all did.  If not, the CTA
// is about to leave, and copies that were only late must have landed before it gives its shared memory back (waited for with a limit).
__device__ __forceinline__ bool all_landed(bool here, bool pending, uint32_t bar, uint32_t parity) {
  if (!__syncthreads_or(!here)) return true;
  int never = 0;
  if (pending) umma::mbar_wait(bar, parity, &never, 1 << 16);
  __syncthreads();
  return false;
}
// The rows of a chunk's nt tokens, `width` columns each; zeros behind them up to `padded` columns and C rows.
__device__ __forceinline__ void copy_rows(uint8_t* dst, int pitch, const __nv_bfloat16* src, int64_t stride, int nt, int width,
                                          int padded, int tid, int threads, uint32_t bar) {
  for (int r = tid; r < C; r += threads) {
    uint8_t* row = dst + r * pitch;
    if (r < nt) copy_piece(row, src + r * stride, width * 2, bar);
    for (int c = r < nt ? width : 0; c < padded; c += 8) *reinterpret_cast<uint4*>(row + c * 2) = make_uint4(0u, 0u, 0u, 0u);
  }
}

// Shared memory of one stage of the scan (elements of bf16, rows padded by 16 bytes)
template <int DK>
struct ScanLayout {
  static constexpr int ROWK = DK + 8;
  int rowv, k, q, v, p, f, bytes;      // byte offsets inside a stage
  __host__ __device__ explicit ScanLayout(int dv) {
    rowv = dv + 8;
    k = 0;
    q = k + C * ROWK * 2;
    v = q + C * ROWK * 2;
    p = v + C * rowv * 2;
    const int staged = C * (dv + 4) * 4;         // outputs are staged over K, Q and V
    if (p < staged) p = staged;
    f = p + 6 * kPlane * 4;
    bytes = f + 4 * C * 4;
  }
};

// ROWS: rows come as bulk copies, else as 16-byte pieces by all threads.  A bulk copy per row is issued by one thread after the other, on
// the warps of the chain, which few warps feel more than they gain: 16 sequences of 1,024 tokens, heads of 128 x 128 589 us in rows and
// 601 in pieces, 128 x 64 312 and 290, 32 x 64 262 and 234, 16 x 16 532 and 458; T, P and the factors, one copy, are a gain at every size.
template <int DK, bool ROWS>
__global__ void __launch_bounds__(256, 1) delta_scan_kernel(const ChunkArgs args) {
  using Lay = ScanLayout<DK>;
  constexpr int ROWK = Lay::ROWK, NK = DK / 8;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ __align__(8) uint64_t s_bars[2];
  __shared__ int s_first;
  __shared__ volatile int s_abort;
  const DeltaArgs& a = args.d;
  const int head = blockIdx.x, seq = blockIdx.y, kh = head / (a.H / a.G), dk = a.dk, dv = a.dv;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3, NT = blockDim.x;
  SeqInfo info;
  if (!sequence_info(a, seq, &info)) return;
  if (tid < 32) {
    const int first = first_segment(a.cu_q, C, seq);
    if (tid == 0) {
      s_first = first;
      s_abort = 0;
      for (int i = 0; i < 2; ++i) umma::mbar_init(smem_u32(&s_bars[i]), 1);
      umma::mbar_init_fence();
    }
  }
  __syncthreads();
  const Lay lay(dv);
  const int chunks = (info.len + C - 1) / C;
  const uint8_t* blob0 = args.blobs + (static_cast<size_t>(s_first) * a.H + head) * kBlobBytes;
  const uint32_t sbase = smem_u32(smem);
  auto bar_of = [&](int j) { return smem_u32(&s_bars[j & 1]); };
  auto fetch = [&](int j) {
    uint8_t* st = smem + (j & 1) * lay.bytes;
    const int nt = min(C, info.len - j * C);
    const int64_t tok = info.tok0 + j * C;
    if (tid == 0) {
      umma::mbar_expect_tx(bar_of(j), (ROWS ? nt * (2 * dk + dv) * 2 : 0) + kBlobBytes);
      copy_piece(st + lay.p, blob0 + static_cast<size_t>(j) * a.H * kBlobBytes, kBlobBytes, bar_of(j));      // T, P, factors
    }
    auto rows = [&](int at, int pitch, const void* src, int off, int width, int padded) {
      const __nv_bfloat16* from = static_cast<const __nv_bfloat16*>(src) + tok * a.act_stride + off;
      if constexpr (ROWS) {
        copy_rows(st + at, pitch, from, a.act_stride, nt, width, padded, tid, NT, bar_of(j));
      } else {
        const int pieces = padded / 8;
        for (int i = tid; i < C * pieces; i += NT) {
          const int r = i / pieces, c = i - r * pieces;
          const bool ok = r < nt && c * 8 < width;
          cp_async16(smem_u32(st + at + r * pitch + c * 16), from + (ok ? r * a.act_stride + c * 8 : 0), ok ? 16 : 0);
        }
      }
    };
    rows(lay.k, ROWK * 2, a.k, kh * dk, dk, DK);
    rows(lay.q, ROWK * 2, a.q, kh * dk, dk, DK);
    rows(lay.v, lay.rowv * 2, a.v, head * dv, dv, dv);
    if constexpr (!ROWS) cp_async_commit();
  };

  // S^T: rows 16 warp + g (+ 8), columns 8 n + 2 tq (+ 1)
  float S[NK][4];
  float* pool = a.state + (info.slot * a.H + head) * static_cast<int64_t>(dk) * dv;
  const int vr = warp * 16 + g;
#pragma unroll
  for (int n = 0; n < NK; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = n * 8 + 2 * tq + (e & 1);
      S[n][e] = !info.fresh && d < dk ? pool[static_cast<int64_t>(d) * dv + vr + 8 * (e >> 1)] : 0.f;
    }

  fetch(0);
  const int r_in = (lane & 7) + (lane >> 4) * 8, bh = (lane >> 3) & 1;      // B operand, rows = n: (n lo, k lo) (n lo, k hi) (n hi, ...)
  const int t_in = (lane & 7) + ((lane >> 3) & 1) * 8, th = lane >> 4;      // B operand transposed, rows = k
  for (int j = 0; j < chunks; ++j) {
    const bool here = umma::mbar_wait(bar_of(j), (j >> 1) & 1, &s_abort);
    if (!here) {
      s_abort = 1;
      report(a.status, B200_ERR_TIMEOUT);
    }
    if constexpr (!ROWS) cp_async_wait<0>();
    umma::fence_async_proxy();                         // outputs were staged where the next copies go
    // chunk j, the only one on its way, has landed; everyone has left the other stage
    if (!all_landed(here, true, bar_of(j), (j >> 1) & 1)) return;
    if (j + 1 < chunks) fetch(j + 1);
    uint8_t* stp = smem + (j & 1) * lay.bytes;
    const uint32_t st = sbase + (j & 1) * lay.bytes;
    const float* f = reinterpret_cast<const float*>(stp + lay.f);
    float D[8][4], O[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) D[n][e] = O[n][e] = 0.f;
    // ---- (K S)^T and (Q S)^T
#pragma unroll
    for (int kk = 0; kk < DK / 16; ++kk) {
      uint32_t h[4], m[4], l[4];
      split_a(S[2 * kk], S[2 * kk + 1], h, m, l);
#pragma unroll
      for (int np = 0; np < 4; np += 2) {
        uint32_t kf[2][4], qf[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          ldmatrix_x4(kf[u], st + lay.k + (((np + u) * 16 + r_in) * ROWK + kk * 16 + bh * 8) * 2);
          ldmatrix_x4(qf[u], st + lay.q + (((np + u) * 16 + r_in) * ROWK + kk * 16 + bh * 8) * 2);
        }
        auto part = [&](const uint32_t (&p)[4]) {        // eight accumulators between two uses of one
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const uint32_t k0[2] = {kf[u][0], kf[u][1]}, k1[2] = {kf[u][2], kf[u][3]};
            const uint32_t q0[2] = {qf[u][0], qf[u][1]}, q1[2] = {qf[u][2], qf[u][3]};
            mma_bf16_16816(D[2 * (np + u)], p, k0);
            mma_bf16_16816(D[2 * (np + u) + 1], p, k1);
            mma_bf16_16816(O[2 * (np + u)], p, q0);
            mma_bf16_16816(O[2 * (np + u) + 1], p, q1);
          }
        };
        part(l);
        part(m);
        part(h);
      }
    }
    // ---- D <- V^T - gamma rk D,  O <- gamma rq O
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      uint32_t vf[4];      // (tokens lo, columns lo) (tokens lo, columns hi) (tokens hi, ...)
      ldmatrix_x4_trans(vf, st + lay.v + ((np * 16 + (lane & 7) + (lane >> 4) * 8) * lay.rowv + warp * 16 + bh * 8) * 2);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int n = 2 * np + u;
        const float2 qs = *reinterpret_cast<const float2*>(f + n * 8 + 2 * tq);
        const float2 ks = *reinterpret_cast<const float2*>(f + C + n * 8 + 2 * tq);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const uint32_t v = vf[2 * u + hh];
          D[n][2 * hh] = __uint_as_float(v << 16) - ks.x * D[n][2 * hh];
          D[n][2 * hh + 1] = __uint_as_float(v & 0xffff0000u) - ks.y * D[n][2 * hh + 1];
          O[n][2 * hh] *= qs.x;
          O[n][2 * hh + 1] *= qs.y;
        }
      }
    }
    // ---- U^T = D^T T^T, then O^T += U^T P^T: B rows are rows of T / P, lower triangle of 16-tiles
    float U[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) U[n][e] = 0.f;
    auto triangular = [&](const float (&in)[8][4], float (&acc)[8][4], int mat) {
      const uint4* base = reinterpret_cast<const uint4*>(stp + lay.p) + mat * 3 * kPlane / 4 + lane;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t h[4], m[4], l[4];
        split_a(in[2 * kk], in[2 * kk + 1], h, m, l);
#pragma unroll
        for (int n0 = kk & ~1; n0 < 4; n0 += 2) {        // two tiles of 16 rows; the first may lie above the diagonal
          uint32_t b3[2][3][4];
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if (n0 + u >= kk) {
#pragma unroll
              for (int p = 0; p < 3; ++p) {
                const uint4 x = base[p * kPlane / 4 + tile_of(n0 + u, kk) * 32];
                b3[u][p][0] = x.x, b3[u][p][1] = x.y, b3[u][p][2] = x.z, b3[u][p][3] = x.w;
              }
            }
          auto part = [&](const uint32_t (&x)[4], int p) {
#pragma unroll
            for (int u = 0; u < 2; ++u)
              if (n0 + u >= kk) {
                const uint32_t b0[2] = {b3[u][p][0], b3[u][p][1]}, b1[2] = {b3[u][p][2], b3[u][p][3]};
                mma_bf16_16816(acc[2 * (n0 + u)], x, b0);
                mma_bf16_16816(acc[2 * (n0 + u) + 1], x, b1);
              }
          };
          part(l, 0);
          part(m, 1);
          part(h, 2);
          part(m, 0);
          part(h, 1);
          part(h, 0);
        }
      }
    };
    triangular(D, U, 0);
    triangular(U, O, 1);
    // ---- S^T = gamma_C S^T + (U rk gamma_C / gamma)^T K
    const float gc = f[3 * C];
#pragma unroll
    for (int n = 0; n < NK; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[n][e] *= gc;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 cs = *reinterpret_cast<const float2*>(f + 2 * C + (2 * kk + u) * 8 + 2 * tq);
        U[2 * kk + u][0] *= cs.x;
        U[2 * kk + u][1] *= cs.y;
        U[2 * kk + u][2] *= cs.x;
        U[2 * kk + u][3] *= cs.y;
      }
      uint32_t h[4], m[4], l[4];
      split_a(U[2 * kk], U[2 * kk + 1], h, m, l);
#pragma unroll
      for (int c = 0; c < NK; c += 8) {
        uint32_t bf[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          ldmatrix_x4_trans(bf[u], st + lay.k + ((kk * 16 + t_in) * ROWK + (c + 2 * u + th) * 8) * 2);
        auto part = [&](const uint32_t (&x)[4]) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t b0[2] = {bf[u][0], bf[u][1]}, b1[2] = {bf[u][2], bf[u][3]};
            mma_bf16_16816(S[c + 2 * u], x, b0);
            mma_bf16_16816(S[c + 2 * u + 1], x, b1);
          }
        };
        part(l);
        part(m);
        part(h);
      }
    }
    // ---- norm over the value columns, output gate
    // a warp takes the tokens warp, warp + NT / 32, ... in groups of eight; the gates of a group are loaded ahead
    const int nt = min(C, info.len - j * C), NW = NT / 32, c = lane * 4;
    const int64_t tok0 = info.tok0 + j * C;
    const __nv_bfloat16* gp = static_cast<const __nv_bfloat16*>(a.gate) + tok0 * a.proj_stride + head * dv + c;
    uint2 gate[8];
    auto load_gates = [&](int t0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int t = t0 + u * NW;
        gate[u] = c < dv && t < nt ? __ldg(reinterpret_cast<const uint2*>(gp + t * a.proj_stride)) : make_uint2(0u, 0u);
      }
    };
    load_gates(warp);
    __syncthreads();                                   // K, Q, V of this stage are done with
    float* so = reinterpret_cast<float*>(stp);
    const int ldo = dv + 4;
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) so[(n * 8 + 2 * tq + (e & 1)) * ldo + vr + 8 * (e >> 1)] = O[n][e];
    __syncthreads();
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < dv) w = make_float4(__ldg(a.norm_w + c), __ldg(a.norm_w + c + 1), __ldg(a.norm_w + c + 2), __ldg(a.norm_w + c + 3));
    for (int t0 = warp; t0 < nt; t0 += 8 * NW) {
      if (t0 != warp) load_gates(t0);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int t = t0 + u * NW;
        if (t >= nt) continue;                         // the same for the whole warp
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < dv) o = *reinterpret_cast<const float4*>(so + t * ldo + c);
        const float inv = rsqrtf(warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w) / static_cast<float>(dv) + a.eps);
        const float2 g0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gate[u].x));
        const float2 g1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gate[u].y));
        using bf16 = __nv_bfloat16;
        if (c < dv)
          *reinterpret_cast<uint2*>(static_cast<bf16*>(a.out) + ((tok0 + t) * a.H + head) * dv + c) =
              make_uint2(pack_bf16x2(o.x * inv * w.x * silu_for<bf16>(g0.x), o.y * inv * w.y * silu_for<bf16>(g0.y)),
                         pack_bf16x2(o.z * inv * w.z * silu_for<bf16>(g1.x), o.w * inv * w.w * silu_for<bf16>(g1.y)));
      }
    }
  }
#pragma unroll
  for (int n = 0; n < NK; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = n * 8 + 2 * tq + (e & 1);
      if (d < dk) pool[static_cast<int64_t>(d) * dv + vr + 8 * (e >> 1)] = S[n][e];
    }
}

// dk = 64, dv <= 64: the same scan by two groups of warps, so that the chain from state to state carries three of the five products
// only.  The scan warps leave the state at a chunk's start and U behind, as their accumulators lie; the output warps, one chunk
// later, make O = diag(gamma rq) Q S + P U of them, norm, gate and store.  One barrier per chunk.
// What bounds it: a scan warp and an output warp share a scheduler, 528 tensor-core products of 8 clocks and the splits between
// them, 8,000 clocks a chunk.  8 prompts of 700 to 1,300 tokens, 8 heads of 64: 100 us; all five products, the epilogue and
// copies by all threads in one chain 197 us.  Heads of 128 stay on the kernel above: both groups do not fit the registers.
struct SplitLayout {
  static constexpr int rows = C * 128;           // K, Q or V: 64 columns, 128-byte swizzle
  static constexpr int k = 0, v = rows, t = 2 * rows, fs = t + 3 * kPlane * 4, scan_bytes = fs + 4 * C * 4;
  static constexpr int q = 0, p = rows, fo = p + 3 * kPlane * 4, out_bytes = fo + 4 * C * 4;
  static constexpr int LDO = 64 + 4;
  static constexpr int out0 = 2 * scan_bytes, hand0 = out0 + 2 * out_bytes;
  static constexpr int hand = 4 * 32 * 32 * 4;   // four warps x 32 words per lane: one state or one U
  static constexpr int so = hand0 + 4 * hand, bytes = so + C * LDO * 4 + 1024;     // 1024: alignment
  static_assert(scan_bytes % 1024 == 0 && out_bytes % 1024 == 0, "tiles of a swizzled copy start on 1024 bytes");
};

__global__ void __launch_bounds__(256, 1) delta_split_kernel(const ChunkArgs args, const __grid_constant__ CUtensorMap tm_q,
                                                             const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v) {
  using Lay = SplitLayout;
  constexpr int NK = 8;
  extern __shared__ __align__(16) uint8_t raw[];
  uint8_t* smem = raw + (-smem_u32(raw) & 1023);
  __shared__ __align__(8) uint64_t s_bars[2][2];   // copies into the stages of the scan, of the outputs
  __shared__ int s_first;
  __shared__ volatile int s_abort;
  const DeltaArgs& a = args.d;
  const int head = blockIdx.x, seq = blockIdx.y, kh = head / (a.H / a.G), dk = a.dk, dv = a.dv;
  const int NT = blockDim.x / 2, tid = threadIdx.x % NT, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
  const bool outputs = threadIdx.x >= NT;
  SeqInfo info;
  if (!sequence_info(a, seq, &info)) return;
  if (threadIdx.x < 32) {
    const int first = first_segment(a.cu_q, C, seq);
    if (threadIdx.x == 0) {
      s_first = first;
      s_abort = 0;
      for (int i = 0; i < 4; ++i) umma::mbar_init(smem_u32(&s_bars[i >> 1][i & 1]), 1);
      umma::mbar_init_fence();
    }
  }
  __syncthreads();
  const int chunks = (info.len + C - 1) / C, vr = warp * 16 + g;
  const uint8_t* blob0 = args.blobs + (static_cast<size_t>(s_first) * a.H + head) * kBlobBytes;
  const int r_in = (lane & 7) + (lane >> 4) * 8, bh = (lane >> 3) & 1;      // B operand, rows = n: (n lo, k lo) (n lo, k hi) (n hi, ...)
  const int t_in = (lane & 7) + ((lane >> 3) & 1) * 8, th = lane >> 4;      // B operand transposed, rows = k
  // 64 columns of a chunk's rows, by one thread; rows behind its tokens are another sequence's and zeroed once they are here
  auto copy_tile = [&](uint8_t* dst, const CUtensorMap& map, int column, int j, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                     smem_u32(dst)), "l"(&map), "r"(column), "r"(static_cast<int>(info.tok0) + j * C), "r"(bar) : "memory");
  };
  // byte offset of eight columns of a row
  auto at_row = [&](int r, int c8) { return r * 128 + ((c8 ^ (r & 7)) << 4); };
  auto bar_of = [&](int j) { return smem_u32(&s_bars[outputs][j & 1]); };
  // chunk j of this half, the only one on its way, has landed, `rows` bytes of rows at `tile`, for every thread of both halves: false
  // if one of them never will
  auto landed = [&](int j, bool wait, uint8_t* tile, int rows) {
    const bool here = !wait || umma::mbar_wait(bar_of(j), (j >> 1) & 1, &s_abort);
    if (!here) {
      s_abort = 1;
      report(a.status, B200_ERR_TIMEOUT);
    }
    const int nt = info.len - j * C;
    if (wait && here && nt < C)
      for (int i = tid; i < rows / 16; i += NT)
        if ((i / 8) % C >= nt) reinterpret_cast<uint4*>(tile)[i] = make_uint4(0u, 0u, 0u, 0u);
    return all_landed(here, wait, bar_of(j), (j >> 1) & 1);
  };
  auto blob_of = [&](int j) { return blob0 + static_cast<size_t>(j) * a.H * kBlobBytes; };
  // this lane's words of a state (0) or U (1) of chunk j
  auto handed = [&](int what, int j) {
    return reinterpret_cast<float4*>(smem + Lay::hand0 + (what * 2 + (j & 1)) * Lay::hand) + warp * 8 * 32 + lane;
  };
  // acc += in T^T or in P^T: B rows are rows of the triangular matrix at `base`
  auto triangular = [&](const float (&in)[8][4], float (&acc)[8][4], const uint8_t* at) {
    const uint4* base = reinterpret_cast<const uint4*>(at) + lane;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t h[4], m[4], l[4];
      split_a(in[2 * kk], in[2 * kk + 1], h, m, l);
#pragma unroll
      for (int n0 = kk & ~1; n0 < 4; n0 += 2) {        // two tiles of 16 rows; the first may lie above the diagonal
        uint4 b3[2][3];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (n0 + u >= kk) {
#pragma unroll
            for (int p = 0; p < 3; ++p) b3[u][p] = base[p * kPlane / 4 + tile_of(n0 + u, kk) * 32];
          }
        auto part = [&](const uint32_t (&x)[4], int p) {
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if (n0 + u >= kk) {
              const uint32_t b0[2] = {b3[u][p].x, b3[u][p].y}, b1[2] = {b3[u][p].z, b3[u][p].w};
              mma_bf16_16816(acc[2 * (n0 + u)], x, b0);
              mma_bf16_16816(acc[2 * (n0 + u) + 1], x, b1);
            }
        };
        part(l, 0);
        part(m, 1);
        part(h, 2);
        part(m, 0);
        part(h, 1);
        part(h, 0);
      }
    }
  };
  // acc += in X^T for the bf16 rows X at `base`, one 16-column step
  auto rows_product = [&](const float (&t0)[4], const float (&t1)[4], float (&acc)[8][4], uint32_t base, int kk) {
    uint32_t h[4], m[4], l[4], bf[4][4];
    split_a(t0, t1, h, m, l);
#pragma unroll
    for (int u = 0; u < 4; ++u) ldmatrix_x4(bf[u], base + at_row(u * 16 + r_in, kk * 2 + bh));
    auto part = [&](const uint32_t (&x)[4]) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t b0[2] = {bf[u][0], bf[u][1]}, b1[2] = {bf[u][2], bf[u][3]};
        mma_bf16_16816(acc[2 * u], x, b0);
        mma_bf16_16816(acc[2 * u + 1], x, b1);
      }
    };
    part(l);
    part(m);
    part(h);
  };

  if (outputs) {
    auto fetch = [&](int j) {
      if (tid != 0) return;
      uint8_t* st = smem + Lay::out0 + (j & 1) * Lay::out_bytes;
      constexpr int bytes = 3 * kPlane * 4 + 4 * C * 4;          // P, then the factors
      umma::mbar_expect_tx(bar_of(j), Lay::rows + bytes);
      copy_tile(st + Lay::q, tm_q, kh * dk, j, bar_of(j));
      copy_piece(st + Lay::p, blob_of(j) + 3 * kPlane * 4, bytes, bar_of(j));
    };
    const int c = (lane & 15) * 4;
    const float4 w = c < dv ? make_float4(__ldg(a.norm_w + c), __ldg(a.norm_w + c + 1), __ldg(a.norm_w + c + 2), __ldg(a.norm_w + c + 3))
                            : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j <= chunks; ++j) {            // outputs of chunk j - 1
      if (!landed(j - 1, j > 0, smem + Lay::out0 + ((j - 1) & 1) * Lay::out_bytes + Lay::q, Lay::rows)) return;
      if (j < chunks) fetch(j);
      if (j == 0) continue;
      const int jj = j - 1, nt = min(C, info.len - jj * C), NW = NT / 32;
      const uint8_t* stp = smem + Lay::out0 + (jj & 1) * Lay::out_bytes;
      const float* f = reinterpret_cast<const float*>(stp + Lay::fo);
      const int64_t tok0 = info.tok0 + jj * C;
      // a half-warp norms the tokens t_own, t_own + 2 NW, ... in groups of eight; the gates of a group are loaded ahead
      const int t_own = 2 * warp + (lane >> 4);
      const __nv_bfloat16* gp = static_cast<const __nv_bfloat16*>(a.gate) + tok0 * a.proj_stride + head * dv + c;
      uint2 gate[8];
      auto load_gates = [&](int t0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int t = t0 + u * 2 * NW;
          gate[u] = c < dv && t < nt ? __ldg(reinterpret_cast<const uint2*>(gp + t * a.proj_stride)) : make_uint2(0u, 0u);
        }
      };
      load_gates(t_own);
      float O[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) O[n][e] = 0.f;
      const float4* hs = handed(0, jj);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const float4 x = hs[2 * kk * 32], y = hs[(2 * kk + 1) * 32];
        const float t0[4] = {x.x, x.y, x.z, x.w}, t1[4] = {y.x, y.y, y.z, y.w};
        rows_product(t0, t1, O, smem_u32(stp) + Lay::q, kk);
      }
      const float4* hu = handed(1, jj);
      float U[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const float2 qs = *reinterpret_cast<const float2*>(f + n * 8 + 2 * tq);
        O[n][0] *= qs.x;
        O[n][1] *= qs.y;
        O[n][2] *= qs.x;
        O[n][3] *= qs.y;
        const float4 x = hu[n * 32];
        U[n][0] = x.x, U[n][1] = x.y, U[n][2] = x.z, U[n][3] = x.w;
      }
      triangular(U, O, stp + Lay::p);
      // ---- norm over the value columns, output gate
      float* so = reinterpret_cast<float*>(smem + Lay::so);
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) so[(n * 8 + 2 * tq + (e & 1)) * Lay::LDO + vr + 8 * (e >> 1)] = O[n][e];
      asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
      for (int t0 = t_own; t0 - (lane >> 4) < nt; t0 += 16 * NW) {
        if (t0 != t_own) load_gates(t0);
        float4 o[8];
        float ss[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {              // eight sums side by side
          const int t = t0 + u * 2 * NW;
          o[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (c < dv && t < nt) o[u] = *reinterpret_cast<const float4*>(so + t * Lay::LDO + c);
          ss[u] = o[u].x * o[u].x + o[u].y * o[u].y + o[u].z * o[u].z + o[u].w * o[u].w;
        }
#pragma unroll
        for (int step = 8; step > 0; step >>= 1)
#pragma unroll
          for (int u = 0; u < 8; ++u) ss[u] += __shfl_xor_sync(0xffffffffu, ss[u], step);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int t = t0 + u * 2 * NW;
          const float inv = rsqrtf(ss[u] / static_cast<float>(dv) + a.eps);
          const float2 g0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gate[u].x));
          const float2 g1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gate[u].y));
          using bf16 = __nv_bfloat16;
          if (c < dv && t < nt)
            *reinterpret_cast<uint2*>(static_cast<bf16*>(a.out) + ((tok0 + t) * a.H + head) * dv + c) =
                make_uint2(pack_bf16x2(o[u].x * inv * w.x * silu_for<bf16>(g0.x), o[u].y * inv * w.y * silu_for<bf16>(g0.y)),
                           pack_bf16x2(o[u].z * inv * w.z * silu_for<bf16>(g1.x), o[u].w * inv * w.w * silu_for<bf16>(g1.y)));
        }
      }
    }
    return;
  }

  // ---- the scan.  S^T: rows 16 warp + g (+ 8), columns 8 n + 2 tq (+ 1)
  auto fetch = [&](int j) {
    if (tid != 0) return;
    uint8_t* st = smem + (j & 1) * Lay::scan_bytes;
    umma::mbar_expect_tx(bar_of(j), Lay::scan_bytes);
    copy_tile(st + Lay::k, tm_k, kh * dk, j, bar_of(j));
    copy_tile(st + Lay::v, tm_v, head * dv, j, bar_of(j));
    copy_piece(st + Lay::t, blob_of(j), 3 * kPlane * 4, bar_of(j));
    copy_piece(st + Lay::fs, blob_of(j) + 6 * kPlane * 4, 4 * C * 4, bar_of(j));
  };
  float S[NK][4];
  float* pool = a.state + (info.slot * a.H + head) * static_cast<int64_t>(dk) * dv;
#pragma unroll
  for (int n = 0; n < NK; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = n * 8 + 2 * tq + (e & 1);
      S[n][e] = !info.fresh && d < dk ? pool[static_cast<int64_t>(d) * dv + vr + 8 * (e >> 1)] : 0.f;
    }
  fetch(0);
  for (int j = 0; j <= chunks; ++j) {
    // everyone has left the buffers of chunk j - 2
    if (!landed(j, j < chunks, smem + (j & 1) * Lay::scan_bytes, 2 * Lay::rows)) return;
    if (j + 1 < chunks) fetch(j + 1);
    if (j == chunks) break;
    const uint8_t* stp = smem + (j & 1) * Lay::scan_bytes;
    const uint32_t st = smem_u32(stp);
    const float* f = reinterpret_cast<const float*>(stp + Lay::fs);
    float4* hs = handed(0, j);
    float D[8][4], U[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      hs[n * 32] = make_float4(S[n][0], S[n][1], S[n][2], S[n][3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) D[n][e] = U[n][e] = 0.f;
    }
    // ---- (K S)^T, then D <- V^T - gamma rk D
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) rows_product(S[2 * kk], S[2 * kk + 1], D, st + Lay::k, kk);
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      uint32_t vf[4];      // (tokens lo, columns lo) (tokens lo, columns hi) (tokens hi, ...)
      ldmatrix_x4_trans(vf, st + Lay::v + at_row(np * 16 + r_in, warp * 2 + bh));
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int n = 2 * np + u;
        const float2 ks = *reinterpret_cast<const float2*>(f + C + n * 8 + 2 * tq);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const uint32_t v = vf[2 * u + hh];
          D[n][2 * hh] = __uint_as_float(v << 16) - ks.x * D[n][2 * hh];
          D[n][2 * hh + 1] = __uint_as_float(v & 0xffff0000u) - ks.y * D[n][2 * hh + 1];
        }
      }
    }
    // ---- U^T = D^T T^T
    triangular(D, U, stp + Lay::t);
    float4* hu = handed(1, j);
    const float gc = f[3 * C];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      hu[n * 32] = make_float4(U[n][0], U[n][1], U[n][2], U[n][3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) S[n][e] *= gc;
    }
    // ---- S^T = gamma_C S^T + (U rk gamma_C / gamma)^T K
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 cs = *reinterpret_cast<const float2*>(f + 2 * C + (2 * kk + u) * 8 + 2 * tq);
        U[2 * kk + u][0] *= cs.x;
        U[2 * kk + u][1] *= cs.y;
        U[2 * kk + u][2] *= cs.x;
        U[2 * kk + u][3] *= cs.y;
      }
      uint32_t h[4], m[4], l[4], bf[4][4];
      split_a(U[2 * kk], U[2 * kk + 1], h, m, l);
#pragma unroll
      for (int u = 0; u < 4; ++u) ldmatrix_x4_trans(bf[u], st + Lay::k + at_row(kk * 16 + t_in, 2 * u + th));
      auto part = [&](const uint32_t (&x)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t b0[2] = {bf[u][0], bf[u][1]}, b1[2] = {bf[u][2], bf[u][3]};
          mma_bf16_16816(S[2 * u], x, b0);
          mma_bf16_16816(S[2 * u + 1], x, b1);
        }
      };
      part(l);
      part(m);
      part(h);
    }
  }
#pragma unroll
  for (int n = 0; n < NK; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = n * 8 + 2 * tq + (e & 1);
      if (d < dk) pool[static_cast<int64_t>(d) * dv + vr + 8 * (e >> 1)] = S[n][e];
    }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

EncodeFn tensor_map_encoder() {
  static const EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found{};
    const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &found) == cudaSuccess &&
                    found == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<EncodeFn>(p) : nullptr;
  }();
  return fn;
}

// tiles of 64 rows x 64 columns of [tokens, columns]
bool tile_map(CUtensorMap* m, const void* base, int64_t tokens, int columns, int64_t stride) {
  const EncodeFn enc = tensor_map_encoder();
  if (enc == nullptr || tokens > 2147483647) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(columns), static_cast<cuuint64_t>(tokens)}, strides[1] = {static_cast<cuuint64_t>(stride) * 2};
  const cuuint32_t box[2] = {64, C}, steps[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline int64_t chunk_count(int num_seqs, int64_t total_tokens) { return total_tokens / C + num_seqs; }

template <int DK>
int launch(const ChunkArgs& c, int64_t total_tokens, cudaStream_t s) {
  const size_t prep = sizeof(PrepSmem<DK>);
  const ScanLayout<DK> lay(c.d.dv);
  const size_t scan = 2 * static_cast<size_t>(lay.bytes);
  constexpr int kRowsFrom = DK == 128 ? 96 : 1 << 30;      // value columns from which rows come as bulk copies
  auto walk = DK == 128 && c.d.dv >= kRowsFrom ? delta_scan_kernel<DK, DK == 128> : delta_scan_kernel<DK, false>;
  if (cudaFuncSetAttribute(delta_prepare_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(prep)) !=
          cudaSuccess ||
      cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(scan)) != cudaSuccess)
    return B200_ERR_LAUNCH;
  delta_prepare_kernel<DK><<<dim3(static_cast<unsigned>(chunk_count(c.d.n, total_tokens)), c.d.H), kPrepThreads, prep, s>>>(c);
  CUtensorMap tq, tk, tv;
  const DeltaArgs& d = c.d;
  if (d.dk == 64 && d.dv <= 64 && tile_map(&tq, d.q, total_tokens, d.G * 64, d.act_stride) &&
      tile_map(&tk, d.k, total_tokens, d.G * 64, d.act_stride) && tile_map(&tv, d.v, total_tokens, d.H * d.dv, d.act_stride)) {
    if (cudaFuncSetAttribute(delta_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitLayout::bytes) != cudaSuccess)
      return B200_ERR_LAUNCH;
    delta_split_kernel<<<dim3(c.d.H, c.d.n), c.d.dv * 4, SplitLayout::bytes, s>>>(c, tq, tk, tv);
  } else {
    walk<<<dim3(c.d.H, c.d.n), c.d.dv * 2, scan, s>>>(c);
  }
  return launch_result();
}

}  // namespace

bool delta_chunk_shape(int dk, int dv) { return dk % 16 == 0 && dv % 16 == 0 && dk <= 128 && dv <= 128; }

size_t delta_chunk_workspace(int num_seqs, int64_t total_tokens, int H) {
  return static_cast<size_t>(chunk_count(num_seqs, total_tokens)) * H * kBlobBytes;
}

int delta_chunk_launch(const DeltaArgs& a, int64_t total_tokens, void* workspace, cudaStream_t s) {
  ChunkArgs c{a, static_cast<uint8_t*>(workspace)};
  return a.dk <= 64 ? launch<64>(c, total_tokens, s) : launch<128>(c, total_tokens, s);
}

}  // namespace b200
