// Gated recurrence of prompts and portions on tensor cores (mathematics and passes: gated_recurrence.cu), sixteen tokens at a time.
// With F_t the product of the forget gates of a block up to token t, F_s,t that of the tokens behind s up to t, and S the state
// at the block's start:
//
//   O = Q~ S + A V,   S' = diag(F_15) S + K~^T V         Q~_t = q_t F_t,   K~_s = k_s F_s,15
//   A_ts = sum_c q_tc k_sc F_s,t,c    s <= t
//
// All factors are products of gates as they stand: nothing is divided and nothing is taken through a logarithm, so a channel
// that forgets everything within a block is as exact as one that keeps it.
//
// One CTA per (segment, head), one barrier per block.  Half of its warps multiply: a warp owns 16 value columns, and S^T [16, D]
// stays in its registers as the accumulators of K~^T V, which have the layout of the next product's A operand.  The other
// half is a block ahead and prepares: gates, Q~ and K~ (a thread owns two channels x four tokens), then A (a warp takes one
// token s and its mirror 15 - s: 17 pairs each, lanes own channels).
//
// Precision: V is bf16 as it comes and exact.  S, Q~, K~ and A are fp32 values split into three bf16 parts that carry 24 bits
// together; products of two of them take the six part products that matter, products with V three; sums are fp32.
//
// What bounds it: issue slots and the latency of a block on sixteen warps per SM (3.5 us a block of D = 128; 1,900 instructions
// a warp).  Both halves in one warp, with two barriers per block, took 549 us where this takes 227 (8 prompts of 1,024 tokens
// x 16 heads x 128 x 128); the scalar walk, 5 FMA per state element and token over two passes, took 786.
//
// Against 64 bits the states are 3.6e-8 .. 1.4e-7 off, the scalar walk's 3.5e-8 .. 1.4e-7.  Long memories (1,024 to 32,768 tokens,
// values of one sign): channels that keep 0.999 per token 1.6e-7 .. 2.4e-7, the walk's 4e-6 .. 1e-5; 0.9999 1.9e-7 .. 4.8e-7, the
// walk's 5e-6 .. 9e-5.  With the state as the accumulator of K~^T V and plain products of gates it was 1.35e-5 and 1.6e-4 (224 us).
#include "recurrence_common.cuh"

namespace b200 {
namespace {

constexpr int BT = 16;                         // tokens per block
constexpr int kOwn = 4;                        // accumulators of K~^T V in flight

// x (two values) -> three packed bf16 pairs whose sum is x to 24 bits
__device__ __forceinline__ void split3(f32x2 x, uint32_t& h, uint32_t& m, uint32_t& l) {
  const f32x2 minus = pack2(-1.f, -1.f);
  float2 y = unpack2(x);
  h = pack_bf16x2(y.x, y.y);
  x = fma2(pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), minus, x);
  y = unpack2(x);
  m = pack_bf16x2(y.x, y.y);
  x = fma2(pack2(__uint_as_float(m << 16), __uint_as_float(m & 0xffff0000u)), minus, x);
  y = unpack2(x);
  l = pack_bf16x2(y.x, y.y);
}
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) { split3(pack2(x0, x1), h, m, l); }

// 1 - (1 - a)(1 - b)
__device__ __forceinline__ float both(float a, float b) { return fmaf(-a, b, a + b); }

template <int D>
struct __align__(16) ChunkSmem {
  static constexpr int ROW = D + 8;            // padded row of the bf16 operands, elements
  static constexpr int ROWA = BT + 8;
  static constexpr int LDO = D + 4;
  __nv_bfloat16 v[2][BT * ROW];
  __nv_bfloat16 k[2][3][BT * ROW];             // parts of K~
  float gamma[2][D];                           // F_15
  __nv_bfloat16 q[2][3][BT * ROW];             // parts of Q~
  __nv_bfloat16 a[2][3][BT * ROWA];            // parts of A, rows t
  float ff[BT * D], kf[BT * D], qf[BT * D];    // gates and queries of a block, columns swizzled by 8 ((t >> 2) & 3)
  float o[BT * LDO];
};

template <int D, bool LOCAL>
__global__ void __launch_bounds__(4 * D, D == 64 ? 2 : 1) recurrence_chunk_kernel(const RecArgs a, const ScanArgs sc) {
  using Sm = ChunkSmem<D>;
  constexpr int NT = 2 * D, NW = NT / 32,          // threads and warps of a half
                 NK = D / 8, ROW = Sm::ROW, ROWA = Sm::ROWA, LDO = Sm::LDO;
  extern __shared__ __align__(16) uint8_t raw[];
  auto half_barrier = [](int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(NT) : "memory"); };
  Sm& sm = *reinterpret_cast<Sm*>(raw);
  const int head = blockIdx.y, number = blockIdx.x;
  int seq, index;
  if (!find_segment(a.cu_q, sc.n, sc.seg_len, number, &seq, &index)) return;
  SeqInfo info;
  if (!sequence_info(a, seq, &info)) return;
  const int segments = (info.len + sc.seg_len - 1) / sc.seg_len;
  const bool last = index == segments - 1;
  if (LOCAL && last) return;                       // its own map is never needed
  const int tok_lo = index * sc.seg_len, ntok = min(sc.seg_len, info.len - tok_lo);
  const int64_t tok0 = info.tok0 + tok_lo;
  const bool ahead = threadIdx.x >= NT;            // the half that prepares
  const int tid = threadIdx.x % NT, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;

  const int blocks = (ntok + BT - 1) / BT;
  if (ahead) {
    // ---- gates of a block: this thread's channels c, c + 1 and tokens 4 tq .. 4 tq + 3
    const int c = (warp * 8 + g) * 2;
    const float2 bias = *reinterpret_cast<const float2*>(a.f_bias + head * D + c);
    const float2 lower = *reinterpret_cast<const float2*>(a.lower + head * D + c);
    const __nv_bfloat16* fp = static_cast<const __nv_bfloat16*>(a.f) + tok0 * a.stride + head * D + c;
    const __nv_bfloat16* qp = static_cast<const __nv_bfloat16*>(a.q) + tok0 * a.stride + head * D + c;
    const __nv_bfloat16* vp = static_cast<const __nv_bfloat16*>(a.v) + tok0 * a.stride + head * D;
    uint32_t rf[4], rq[4];
    auto fetch = [&](int b) {                        // projections of block b -> registers
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = b * BT + tq * 4 + i;
        rf[i] = rq[i] = 0u;
        if (t < ntok) {
          rf[i] = __ldg(reinterpret_cast<const uint32_t*>(fp + t * a.stride));
          if (!LOCAL) rq[i] = __ldg(reinterpret_cast<const uint32_t*>(qp + t * a.stride));
        }
      }
    };
    auto fetch_v = [&](int b) {
      for (int i = tid; i < BT * (D / 8); i += NT) {
        const int r = i / (D / 8), cc = i % (D / 8), t = b * BT + r;
        cp_async16(smem_u32(&sm.v[b & 1][r * ROW + cc * 8]), vp + (t < ntok ? t * a.stride + cc * 8 : 0), t < ntok ? 16 : 0);
      }
      cp_async_commit();
    };
    float dec = 1.f, owed = 0.f;                     // of channel c + (tq & 1): product of the segment's gates; see below
    auto gate_block = [&](int b) {
      float f[4][2], k[4][2], q[4][2];
      const int sw = c ^ (tq * 8);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool ok = b * BT + tq * 4 + i < ntok;
        gates(__uint_as_float(rf[i] << 16) + bias.x, lower.x, &f[i][0], &k[i][0]);
        gates(__uint_as_float(rf[i] & 0xffff0000u) + bias.y, lower.y, &f[i][1], &k[i][1]);
        if (!ok) f[i][0] = f[i][1] = 1.f, k[i][0] = k[i][1] = 0.f;
        if (!LOCAL) {
          q[i][0] = silu_f(__uint_as_float(rq[i] << 16));
          q[i][1] = silu_f(__uint_as_float(rq[i] & 0xffff0000u));
          const int at = (tq * 4 + i) * D + sw;
          *reinterpret_cast<float2*>(sm.ff + at) = make_float2(f[i][0], f[i][1]);
          *reinterpret_cast<float2*>(sm.kf + at) = make_float2(k[i][0], k[i][1]);
          *reinterpret_cast<float2*>(sm.qf + at) = make_float2(q[i][0], q[i][1]);
        }
      }
      float before[2], behind[2], all[2], loss[2];   // products of the other threads' tokens and of all; 1 - product of the own
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float own = (f[0][j] * f[1][j]) * (f[2][j] * f[3][j]);
        float up = own, y = __shfl_up_sync(0xffffffffu, up, 1, 4);
        if (tq >= 1) up *= y;
        y = __shfl_up_sync(0xffffffffu, up, 2, 4);
        if (tq >= 2) up *= y;
        y = __shfl_up_sync(0xffffffffu, up, 1, 4);
        before[j] = tq >= 1 ? y : 1.f;
        float dn = own;
        y = __shfl_down_sync(0xffffffffu, dn, 1, 4);
        if (tq <= 2) dn *= y;
        y = __shfl_down_sync(0xffffffffu, dn, 2, 4);
        if (tq <= 1) dn *= y;
        y = __shfl_down_sync(0xffffffffu, dn, 1, 4);
        behind[j] = tq <= 2 ? y : 1.f;
        all[j] = tq == 3 ? up : dn * before[j];
        loss[j] = both(both(k[0][j], k[1][j]), both(k[2][j], k[3][j]));
      }
      auto put = [&](__nv_bfloat16 (&dst)[3][BT * ROW], int t, float x0, float x1) {
        uint32_t h, m, l;
        split3(x0, x1, h, m, l);
        *reinterpret_cast<uint32_t*>(&dst[0][t * ROW + c]) = h;
        *reinterpret_cast<uint32_t*>(&dst[1][t * ROW + c]) = m;
        *reinterpret_cast<uint32_t*>(&dst[2][t * ROW + c]) = l;
      };
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        before[0] *= f[i][0];
        before[1] *= f[i][1];
        if (!LOCAL) put(sm.q[b & 1], tq * 4 + i, q[i][0] * before[0], q[i][1] * before[1]);
      }
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        put(sm.k[b & 1], tq * 4 + i, k[i][0] * behind[0], k[i][1] * behind[1]);
        behind[0] *= f[i][0];
        behind[1] *= f[i][1];
      }
      // F_15.  Gates just below one round to a product that is always too small, (1 - e)(1 - e') losing an e e' of less than half
      // a step: block after block that would be a decay of its own.  There F_15 is 1 - loss, loss from the write gates 1 - f, and
      // makes up for what the rounding of the block before took (`owed`, relative; 2 - F stands for 1 / F near one).
      {
        const bool odd = tq & 1;
        const float y = __shfl_xor_sync(0xffffffffu, odd ? loss[0] : loss[1], 1), two = both(odd ? loss[1] : loss[0], y);
        const float gone = both(two, __shfl_xor_sync(0xffffffffu, two, 2));
        float gamma = odd ? all[1] : all[0];
        const bool near_one = fabsf(gone) < 0.25f;
        const float x = 1.f - gone, more = fmaf(x, owed, 1.f - x - gone);
        gamma = near_one ? x + more : gamma;
        owed = near_one ? (x - gamma + more) * (2.f - gamma) : 0.f;
        if (LOCAL) dec *= gamma;
        if (tq >= 2) sm.gamma[b & 1][c + odd] = gamma;
      }
    };

    // ---- A of a block: columns s and 15 - s, lanes own CPL channels
    auto scores = [&](int b) {
      constexpr int CPL = D / 32, P = CPL / 2;
      auto at = [&](int t) { return t * D + ((lane * CPL) ^ (((t >> 2) & 3) * 8)); };
      auto load = [&](const float* base, int t, f32x2 (&x)[P]) {
        if constexpr (P == 2) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(base + at(t));
          x[0] = y.x, x[1] = y.y;
        } else {
          x[0] = *reinterpret_cast<const f32x2*>(base + at(t));
        }
      };
      auto dot = [&](const f32x2 (&x)[P], const f32x2 (&y)[P]) {
        f32x2 s = mul2(x[0], y[0]);
        if constexpr (P == 2) s = fma2(x[1], y[1], s);
        const float2 h = unpack2(s);
        return h.x + h.y;
      };
#pragma unroll 1
      for (int s1 = warp; s1 < BT / 2; s1 += NW) {
        const int s2 = BT - 1 - s1;
        f32x2 w1[P], w2[P], f[P], q[P];
        load(sm.kf, s1, w1);
        load(sm.kf, s2, w2);
        float p1[BT], p2[BT / 2];
#pragma unroll
        for (int t = 0; t < BT / 2; ++t) {
          p1[t] = 0.f;
          if (t >= s1) {                             // the same for the whole warp
            load(sm.qf, t, q);
            if (t > s1) {
              load(sm.ff, t, f);
#pragma unroll
              for (int i = 0; i < P; ++i) w1[i] = mul2(w1[i], f[i]);
            }
            p1[t] = dot(q, w1);
          }
        }
#pragma unroll
        for (int t = BT / 2; t < BT; ++t) {
          load(sm.qf, t, q);
          load(sm.ff, t, f);
#pragma unroll
          for (int i = 0; i < P; ++i) w1[i] = mul2(w1[i], f[i]);
          p1[t] = dot(q, w1);
          p2[t - BT / 2] = 0.f;
          if (t >= s2) {
            if (t > s2)
#pragma unroll
              for (int i = 0; i < P; ++i) w2[i] = mul2(w2[i], f[i]);
            p2[t - BT / 2] = dot(q, w2);
          }
        }
        // sums over the lanes; every step a lane keeps half of the rows it still has: row lane >> 1 of p1, 8 + (lane >> 2) of p2
#pragma unroll
        for (int half = BT / 2, step = 16; half >= 1; half >>= 1, step >>= 1) {
          const bool up = lane & step;
#pragma unroll
          for (int i = 0; i < half; ++i) {
            const float send = up ? p1[i] : p1[i + half], keep = up ? p1[i + half] : p1[i];
            p1[i] = keep + __shfl_xor_sync(0xffffffffu, send, step);
          }
        }
        p1[0] += __shfl_xor_sync(0xffffffffu, p1[0], 1);
#pragma unroll
        for (int half = BT / 4, step = 16; half >= 1; half >>= 1, step >>= 1) {
          const bool up = lane & step;
#pragma unroll
          for (int i = 0; i < half; ++i) {
            const float send = up ? p2[i] : p2[i + half], keep = up ? p2[i + half] : p2[i];
            p2[i] = keep + __shfl_xor_sync(0xffffffffu, send, step);
          }
        }
        p2[0] += __shfl_xor_sync(0xffffffffu, p2[0], 2);
        p2[0] += __shfl_xor_sync(0xffffffffu, p2[0], 1);
        uint32_t part[3];
        split3(p1[0], p2[0], part[0], part[1], part[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          if ((lane & 1) == 0) sm.a[b & 1][i][(lane >> 1) * ROWA + s1] = __ushort_as_bfloat16(part[i] & 0xffffu);
          if ((lane & 3) == 0) sm.a[b & 1][i][(BT / 2 + (lane >> 2)) * ROWA + s2] = __ushort_as_bfloat16(part[i] >> 16);
        }
      }
    };

    if constexpr (!LOCAL)                          // above the diagonal A stays zero
      for (int i = tid; i < static_cast<int>(sizeof(sm.a) / 4); i += NT) reinterpret_cast<uint32_t*>(sm.a)[i] = 0u;
    fetch(0);
    for (int b = 0; b <= blocks; ++b) {            // prepares block b while block b - 1 is multiplied
      if (b < blocks) {
        fetch_v(b);
        gate_block(b);
        fetch(b + 1);
        if constexpr (!LOCAL) {
          half_barrier(1);
          scores(b);
        }
        cp_async_wait<0>();
      }
      __syncthreads();
    }
    if (LOCAL && tq >= 2) sc.seg_decay[(static_cast<int64_t>(number) * a.H + head) * D + c + (tq & 1)] = dec;
    return;
  }

  // ---- S^T: rows vr (+ 8), columns 8 n + 2 tq (+ 1)
  float S[NK][4];
  const int64_t head_state = static_cast<int64_t>(D) * D;
  float* pool = a.state + (info.slot * a.H + head) * head_state;
  float* mine = sc.seg_state + (static_cast<int64_t>(number) * a.H + head) * head_state;
  const float* from = LOCAL ? nullptr : segments > 1 ? mine : info.fresh ? nullptr : pool;
  const int vr = warp * 16 + g;
#pragma unroll
  for (int n = 0; n < NK; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      S[n][e] = from != nullptr ? from[(n * 8 + 2 * tq + (e & 1)) * D + vr + 8 * (e >> 1)] : 0.f;

  // ---- norm and store of a block's outputs: a thread takes eight columns of token tid / (D / 8)
  auto store_block = [&](int b) {
    constexpr int TPT = D / 8;                     // threads per token
    const int t = tid / TPT, col = tid % TPT * 8;
    const float4 x = *reinterpret_cast<const float4*>(sm.o + t * LDO + col), y = *reinterpret_cast<const float4*>(sm.o + t * LDO + col + 4);
    float ss = (x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w) + (y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w);
#pragma unroll
    for (int o = TPT / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (b * BT + t >= ntok) return;
    const float inv = rsqrtf(ss / static_cast<float>(D) + a.eps);
    const float4 w0 = __ldg(reinterpret_cast<const float4*>(a.norm_w + col)), w1 = __ldg(reinterpret_cast<const float4*>(a.norm_w + col + 4));
    *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.out) + ((tok0 + b * BT + t) * a.H + head) * D + col) =
        make_uint4(pack_bf16x2(x.x * inv * w0.x, x.y * inv * w0.y), pack_bf16x2(x.z * inv * w0.z, x.w * inv * w0.w),
                   pack_bf16x2(y.x * inv * w1.x, y.y * inv * w1.y), pack_bf16x2(y.z * inv * w1.z, y.w * inv * w1.w));
  };

  // ---- the products of a block
  const int r_in = (lane & 7) + (lane >> 4) * 8, bh = (lane >> 3) & 1;      // B operand, rows = n: (n lo, k lo) (n lo, k hi) (n hi, ...)
  const int t_in = (lane & 7) + ((lane >> 3) & 1) * 8, th = lane >> 4;      // B operand transposed, rows = k
  auto products = [&](int b) {
    const int st = b & 1;
    uint32_t vf[4];
    ldmatrix_x4_trans(vf, smem_u32(&sm.v[st][((lane & 7) + (lane >> 4) * 8) * ROW + warp * 16 + bh * 8]));
    if constexpr (!LOCAL) {
      float O[3][2][4];                            // by the order of the part products: three chains per eight tokens
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) O[i][0][e] = O[i][1][e] = 0.f;
      auto mul = [&](int i, const uint32_t (&x)[4], const uint32_t (&y)[4]) {
        const uint32_t y0[2] = {y[0], y[1]}, y1[2] = {y[2], y[3]};
        mma_bf16_16816(O[i][0], x, y0);
        mma_bf16_16816(O[i][1], x, y1);
      };
#pragma unroll
      for (int kk = 0; kk < NK / 2; ++kk) {
        uint32_t x[3][4], y[3][4];
#pragma unroll
        for (int i = 0; i < 3; ++i) ldmatrix_x4(y[i], smem_u32(&sm.q[st][i][r_in * ROW + kk * 16 + bh * 8]));
        split3(S[2 * kk][0], S[2 * kk][1], x[0][0], x[1][0], x[2][0]);
        split3(S[2 * kk][2], S[2 * kk][3], x[0][1], x[1][1], x[2][1]);
        split3(S[2 * kk + 1][0], S[2 * kk + 1][1], x[0][2], x[1][2], x[2][2]);
        split3(S[2 * kk + 1][2], S[2 * kk + 1][3], x[0][3], x[1][3], x[2][3]);
        mul(2, x[2], y[0]);
        mul(1, x[1], y[0]);
        mul(0, x[0], y[0]);
        mul(2, x[1], y[1]);
        mul(1, x[0], y[1]);
        mul(2, x[0], y[2]);
      }
      bool odd = false;                            // a value that is not finite: it must not meet A's zeros of the tokens before it
#pragma unroll
      for (int i = 0; i < 4; ++i) odd |= (vf[i] & 0x7f80u) == 0x7f80u || (vf[i] & 0x7f800000u) == 0x7f800000u;
      if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = n * 8 + 2 * tq + (e & 1), col = vr + 8 * (e >> 1);
            float sum = 0.f;
#pragma unroll 1
            for (int s = 0; s <= t; ++s) {
              const int at = t * ROWA + s;
              const float w = (__bfloat162float(sm.a[st][2][at]) + __bfloat162float(sm.a[st][1][at])) + __bfloat162float(sm.a[st][0][at]);
              sum += w * __bfloat162float(sm.v[st][s * ROW + col]);
            }
            O[0][n][e] += sum;
          }
      } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          uint32_t y[4];
          ldmatrix_x4(y, smem_u32(&sm.a[st][i][r_in * ROWA + bh * 8]));
          mul(i, vf, y);
        }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          sm.o[(n * 8 + 2 * tq + (e & 1)) * LDO + vr + 8 * (e >> 1)] = (O[2][n][e] + O[1][n][e]) + O[0][n][e];
    }
    // S^T <- diag(gamma) S^T + (K~^T V)^T, the product in accumulators of its own: a tensor core cuts the low bits of the sums it adds
    // to, always to one side, and a state that keeps 0.999 of itself per token would carry the cuts of a thousand tokens
#pragma unroll
    for (int n0 = 0; n0 < NK; n0 += kOwn) {
      float P[kOwn][4];
#pragma unroll
      for (int n = 0; n < kOwn; ++n) P[n][0] = P[n][1] = P[n][2] = P[n][3] = 0.f;
#pragma unroll
      for (int i = 2; i >= 0; --i)
#pragma unroll
        for (int n = 0; n < kOwn; n += 2) {
          uint32_t y[4];
          ldmatrix_x4_trans(y, smem_u32(&sm.k[st][i][t_in * ROW + (n0 + n + th) * 8]));
          const uint32_t y0[2] = {y[0], y[1]}, y1[2] = {y[2], y[3]};
          mma_bf16_16816(P[n], vf, y0);
          mma_bf16_16816(P[n + 1], vf, y1);
        }
#pragma unroll
      for (int n = 0; n < kOwn; ++n) {
        float (&x)[4] = S[n0 + n];
        const f32x2 f = *reinterpret_cast<const f32x2*>(sm.gamma[st] + (n0 + n) * 8 + 2 * tq);
        const float2 u = unpack2(fma2(pack2(x[0], x[1]), f, pack2(P[n][0], P[n][1])));
        const float2 w = unpack2(fma2(pack2(x[2], x[3]), f, pack2(P[n][2], P[n][3])));
        x[0] = u.x, x[1] = u.y, x[2] = w.x, x[3] = w.y;
      }
    }
  };

  __syncthreads();
  for (int b = 0; b < blocks; ++b) {
    products(b);
    if constexpr (!LOCAL) {
      half_barrier(2);
      store_block(b);
    }
    __syncthreads();                               // block b's operands may be overwritten, those of b + 1 are ready
  }
  float* to = LOCAL ? mine : last ? pool : nullptr;
  if (to != nullptr)
#pragma unroll
    for (int n = 0; n < NK; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) to[(n * 8 + 2 * tq + (e & 1)) * D + vr + 8 * (e >> 1)] = S[n][e];
}

template <int D>
int launch(const RecArgs& a, const ScanArgs& sc, int64_t segments, bool chained, cudaStream_t s) {
  constexpr int smem = sizeof(ChunkSmem<D>);
  static bool configured[64] = {false};       // racing threads set the same attributes
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    if (cudaFuncSetAttribute(recurrence_chunk_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaFuncSetAttribute(recurrence_chunk_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return B200_ERR_LAUNCH;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  // segments of uncut sequences are the sequences: no CTA without work in the middle of the grid
  const dim3 grid(static_cast<unsigned>(chained ? segments : sc.n), a.H);
  if (chained) {
    recurrence_chunk_kernel<D, true><<<grid, 4 * D, smem, s>>>(a, sc);
    const int rc = recurrence_chain_launch(a, sc, s);
    if (rc != B200_OK) return rc;
  }
  recurrence_chunk_kernel<D, false><<<grid, 4 * D, smem, s>>>(a, sc);
  return launch_result();
}

}  // namespace

// For sequences that the scan would not cut.  A block costs the same for one token as for sixteen.  In one wave of CTAs the longest
// sequence sets the time (16 x 16 heads of 64: 3 tokens 7.7 us, token by token 6.5; 6 tokens 7.8 and 9.2); above that the rates of both
// count, in ns per sequence and block or token from 1 to 256 sequences of 2 to 33 tokens (256 x 16 heads of 64: 5 tokens 99 us, token by
// token 68; 16 tokens 104 and 120; of 128: 5 tokens 240 and 190, 16 tokens 247 and 338).
bool recurrence_chunk_pays(int n, int64_t total_tokens, int max_seqlen_q, int H, int D) {
  const int sms = sm_count_cached();
  if (static_cast<int64_t>(n) * H <= (D == 64 ? 2 : 1) * static_cast<int64_t>(sms > 0 ? sms : 148)) return max_seqlen_q >= 5;
  const double tokens = static_cast<double>(total_tokens) / n, blocks = max_seqlen_q <= BT ? 1 : static_cast<int64_t>((tokens + BT - 1) / BT);
  return D == 64 ? 12.9 + 10.5 * blocks < 9.5 + 1.23 * tokens : 35.3 + 22.3 * blocks < 29.5 + 3.3 * tokens;
}

int recurrence_chunk_seg_len(int64_t total_tokens, int max_seqlen_q, int H) {
  // one CTA per SM and head; whole sequences as long as the longest takes less than two such shares, since cutting costs
  // two more launches, half of the work again and three passes over the states
  const int64_t share = (total_tokens * H / sm_count_cached() + BT - 1) / BT * BT;
  if (max_seqlen_q <= 2 * share) return static_cast<int>((static_cast<int64_t>(max_seqlen_q) + BT - 1) / BT * BT);
  return static_cast<int>(share < 64 ? 64 : share);
}

int recurrence_chunk_launch(const RecArgs& a, const ScanArgs& sc, int64_t segments, bool chained, cudaStream_t s) {
  return a.dk == 64 ? launch<64>(a, sc, segments, chained, s) : launch<128>(a, sc, segments, chained, s);
}

}  // namespace b200
