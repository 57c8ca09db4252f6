// Chunk-parallel form of the linear recurrences with a decay per key channel and token on warp-level tensor products, for prompts in
// bf16 mode: the gated delta rule (RecurArgs mode 1) and gated linear attention (mode 2 with log_c).  The chunked mathematics is that
// of "Gated Linear Attention Transformers with Hardware-Efficient Training" (Yang et al., 2023) and, for the delta rule's triangular
// system, "Parallelizing Linear Transformers with the Delta Rule over Sequence Length" (Yang et al., 2024).
//
//   S_t = diag(g_t) S_(t-1) + k_t u_t^T,   o_t = S_t^T q_t,   u_t = v_t, or with the delta rule beta_t (v_t - (diag(g_t) S_(t-1))^T k_t)
//
// With c_t the running sum of log g inside a chunk of 64 tokens that starts from the state P:
//   o_t = P^T (q_t e^(c_t)) + sum_{j <= t} B_tj u_j,   B_tj = sum_d q_t k_j e^(c_t - c_j)       (d: key channels)
//   the chunk leaves  diag(e^(c_C)) P + sum_j (k_j e^(c_C - c_j)) u_j^T
//   delta rule:  (I + diag(beta) A) U = diag(beta) (V - (K e^c) P),   A_tj = sum_d k_t k_j e^(c_t - c_j) for j < t,
//   so  U = U' - W P  with  T = (I + diag(beta) A)^-1,  U' = T diag(beta) V,  W = T diag(beta) (K e^c)
//  1. channel_chunk_kernel  a CTA per (chunk, head, sequence), none waits for another: B, A, T, W, U', the decayed queries and keys,
//                           written to the workspace in the order in which the lanes of kernel 2 read them as MMA operands
//  2. channel_chain_kernel  a CTA per (16 value columns, head, sequence) walks the chunks: S^T (16 x DK) stays in fp32 accumulator
//                           registers - a warp owns 16 key channels -, which are the left operand of the next product without a
//                           move.  Per chunk two products against S (W and the decayed queries), a sum over the warps through shared
//                           memory, then the state's and the outputs' products with U; operand blocks are fetched a chunk ahead.
// Every exponential has an argument <= 0: c is kept relative to blocks of 16 tokens, products between blocks take a reference
// between them (e^(c_t - ref) e^(ref - c_j)), 8 x 8 blocks on the diagonal are formed pair by pair.  All operands of the tensor
// products - keys, queries, scores, T, U and the state - are pairs hi + lo of bf16 values (right to 2^-18), a product is
// hi hi + hi lo + lo hi with fp32 accumulation; the inverse is fp32.  The chain these prompts took before keeps them in fp32: alone, a
// layer's outputs are within 2^-15 of 64-bit ones here and within 2^-19 there; the logits, whose projections read bf16, are as far from
// 64-bit ones either way (new over old, 8 seeds each: delta rule 1.0012 +- 0.0022 and 0.9992 +- 0.0018, gated linear attention
// 1.0028 +- 0.0016, all three layers of that family 0.9945 +- 0.0022).  L3_RECUR_CHUNK=0 keeps the chain.
#include <stdint.h>
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"
#include "mixer.h"

namespace {

constexpr int CT = 64;   // tokens per chunk

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&t);
}
// (a, b) as bf16 pairs: hi + lo = value up to 2^-17 of it
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack2(a, b);
  lo = pack2(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += (ah + al) (b.hi + b.lo); b = (hi b0, hi b1, lo b0, lo b1)
__device__ __forceinline__ void mma3(float (&c)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4], const uint4& b) {
  mma16816(c, ah, b.x, b.y);
  mma16816(c, al, b.x, b.y);
  mma16816(c, ah, b.z, b.w);
}

// One (chunk, head, sequence) of the workspace, in 16-byte units: operand blocks W and decayed queries [token tile 8][k step DK / 16]
// [lane], decayed keys [channel tile DK / 8][k step 4][lane], B [token tile 8][k step 4][lane], then e^(c_C) and U' as floats
template <int DK> struct Ws {
  static constexpr int W = 8 * (DK / 16) * 32, Q = W, K = (DK / 8) * 4 * 32, B = 8 * 4 * 32, E = DK / 4;
  static constexpr int oQ = W, oK = oQ + Q, oB = oK + K, oE = oB + B, oU = oE + E;
  __host__ __device__ static size_t total(int DV, bool delta) { return (size_t)oU + (delta ? (size_t)CT * DV / 4 : 0); }
};

// ---------------------------------------------------------------------------------------------- 1. what a chunk needs by itself
// One CTA per SM (104 KB of rows), bound by its own latencies: ~55000 cycles when every product took its exponentials anew from running
// sums and values came one load at a time, of which 13500 went to the tiles between blocks, 7500 to the operands and up to 28000 to the
// values' product.  Now what looks across a block's edge reads rows that are decayed once, in place - queries and keys from the block's
// start, keys to its end -, and the blocks' totals enter as factors per channel.  2048 tokens, 16 heads of 128 x 128: 152 -> 86 us;
// 3 x 701 tokens, 8 heads of 128 x 256 without the delta rule: 37 -> 26.
template <int DK> constexpr int chunk_floats(bool delta) {
  return 3 * CT * (DK + 8) + CT * (CT + 4) + 14 * DK + 2048 + (delta ? 2 * CT * (CT + 4) + 3 * 16 * 17 + CT : 0);
}

template <int DK, bool DELTA>
__global__ void __launch_bounds__(512) channel_chunk_kernel(RecurArgs a, int c0) {
  extern __shared__ __align__(16) float sm[];
  constexpr int LD = DK + 8, LDA = CT + 4;
  float* qf = sm;                       // [CT][LD] queries; later decayed from the start of the block of 16 tokens
  float* kf = qf + CT * LD;             // keys, likewise
  float* lf = kf + CT * LD;             // running log decay inside a block, token included; later keys decayed to the end of the block
  float* Bm = lf + CT * LD;             // [CT][LDA]
  float* tot = Bm + CT * LDA;           // [4][DK] the blocks' totals
  float* fac = tot + 4 * DK;            // [10][DK] decays over whole blocks: 0 | 0 1 | 0 1 2 | all | 1 2 3 | 2 3 | 3 | 1 | 1 2 | 2
  float* part = fac + 10 * DK;          // [quarter of the channels][block][16][8]
  float* Am = part + 2048;              // [CT][LDA] diag(beta) A, strictly lower (delta rule, as what follows)
  float* Tm = Am + CT * LDA;            // [CT][LDA]
  float* tmp = Tm + CT * LDA;           // [3][16][17]
  float* beta = tmp + 3 * 16 * 17;      // [CT]
  pdl_launch();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q2 = (lane & 3) * 2;
  const int c = c0 + blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int n = min(CT, a.L - c * CT);
  const size_t row0 = (size_t)b * a.L + (size_t)c * CT;
  constexpr int IT = CT * DK / 4 / 512;  // 16-byte pieces of a thread
  {
    const float* qs = a.q + row0 * a.ld_q + (size_t)(h / a.rep) * DK;
    const float* ks = a.k + row0 * a.ld_k + (size_t)(h / a.rep) * DK;
    const float* ls = a.log_c + row0 * a.H * DK + (size_t)h * DK;
    float4 qv[IT], kv[IT], lv[IT];
#pragma unroll
    for (int u = 0; u < IT; ++u) {       // all in flight; rows behind the last token read it again and count as zero
      const int i = tid + u * 512, t = min(i / (DK / 4), n - 1), d = (i % (DK / 4)) * 4;
      qv[u] = *reinterpret_cast<const float4*>(qs + (size_t)t * a.ld_q + d);
      kv[u] = *reinterpret_cast<const float4*>(ks + (size_t)t * a.ld_k + d);
      lv[u] = *reinterpret_cast<const float4*>(ls + (size_t)t * a.H * DK + d);
    }
    if (DELTA && tid < CT) beta[tid] = tid < n ? a.beta[(row0 + tid) * a.H + h] : 0.f;
    for (int i = tid; i < CT * LDA; i += 512) { Bm[i] = 0.f; if (DELTA) Am[i] = 0.f; }
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int i = tid + u * 512, t = i / (DK / 4), d = (i % (DK / 4)) * 4;
      float4 l = lv[u];
      // From -104 on a decay is zero in fp32.  Stronger ones are held at -110: the decays of the tokens behind them are differences
      // of running sums, which are right to 2^-14 of a unit that way (a block's stay above -16 x 110), with one such token to 2^-18
      l.x = l.x < -110.f ? -110.f : l.x; l.y = l.y < -110.f ? -110.f : l.y; l.z = l.z < -110.f ? -110.f : l.z; l.w = l.w < -110.f ? -110.f : l.w;
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(qf + t * LD + d) = t < n ? qv[u] : z;
      *reinterpret_cast<float4*>(kf + t * LD + d) = t < n ? kv[u] : z;
      *reinterpret_cast<float4*>(lf + t * LD + d) = t < n ? l : z;
    }
  }
  __syncthreads();
  for (int i = tid; i < 4 * DK; i += 512) {
    const int blk = i / DK, d = i % DK;
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) { s += lf[(blk * 16 + r) * LD + d]; lf[(blk * 16 + r) * LD + d] = s; }
    tot[i] = s;
  }
  __syncthreads();
  // ---- between the halves of a block: tokens 8 - 15 against keys 0 - 7, the reference ahead of the second half; A in the upper rows of
  // the tile, B in the lower ones, a quarter of the channels per warp
  {
    const int I = warp >> 2, kq = warp & 3, t = 16 * I + 8 + g, j = 16 * I + g;
    float acc[4] = {};
#pragma unroll
    for (int k0 = kq * (DK / 4); k0 < (kq + 1) * (DK / 4); k0 += 16) {
      uint32_t ah[4], al[4];
      uint4 bb;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int d = k0 + q2 + 8 * s;
        const float2 ref = *reinterpret_cast<const float2*>(lf + (16 * I + 7) * LD + d);
        const float2 lt = *reinterpret_cast<const float2*>(lf + t * LD + d), lj = *reinterpret_cast<const float2*>(lf + j * LD + d);
        const float2 kt = *reinterpret_cast<const float2*>(kf + t * LD + d), qt = *reinterpret_cast<const float2*>(qf + t * LD + d);
        const float2 kj = *reinterpret_cast<const float2*>(kf + j * LD + d);
        const float ex = __expf(lt.x - ref.x), ey = __expf(lt.y - ref.y);
        split2(kt.x * ex, kt.y * ey, ah[2 * s], al[2 * s]);
        split2(qt.x * ex, qt.y * ey, ah[2 * s + 1], al[2 * s + 1]);
        uint32_t hi, lo;
        split2(kj.x * __expf(ref.x - lj.x), kj.y * __expf(ref.y - lj.y), hi, lo);
        if (s) { bb.y = hi; bb.w = lo; } else { bb.x = hi; bb.z = lo; }
      }
      mma3(acc, ah, al, bb);
    }
    float* o = part + (kq * 4 + I) * 128 + g * 8 + q2;
    *reinterpret_cast<float2*>(o) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(o + 64) = make_float2(acc[2], acc[3]);
  }
  // ---- the 8 x 8 blocks on the diagonal, pair by pair: lane = (token, one of four keys)
  {
    const int t = (warp >> 1) * 8 + g, j = (warp >> 1) * 8 + (warp & 1) * 4 + (lane & 3);
    float sa = 0.f, sb = 0.f;
#pragma unroll 4
    for (int d = 0; d < DK; d += 4) {
      const float4 lt = *reinterpret_cast<const float4*>(lf + t * LD + d), lj = *reinterpret_cast<const float4*>(lf + j * LD + d);
      const float4 kj = *reinterpret_cast<const float4*>(kf + j * LD + d), qt = *reinterpret_cast<const float4*>(qf + t * LD + d);
      const float ex = kj.x * __expf(lt.x - lj.x), ey = kj.y * __expf(lt.y - lj.y), ez = kj.z * __expf(lt.z - lj.z), ew = kj.w * __expf(lt.w - lj.w);
      sb = fmaf(qt.x, ex, sb); sb = fmaf(qt.y, ey, sb); sb = fmaf(qt.z, ez, sb); sb = fmaf(qt.w, ew, sb);
      if (DELTA) {
        const float4 kt = *reinterpret_cast<const float4*>(kf + t * LD + d);
        sa = fmaf(kt.x, ex, sa); sa = fmaf(kt.y, ey, sa); sa = fmaf(kt.z, ez, sa); sa = fmaf(kt.w, ew, sa);
      }
    }
    if (j <= t) Bm[t * LDA + j] = sb;                    // a key behind the query has a positive exponent: never stored
    if (DELTA && j < t) Am[t * LDA + j] = sa * beta[t];
  }
  __syncthreads();
  // ---- the halves' products; rows decayed in place; decays over whole blocks
  {
    const int I = tid >> 7, r = (tid >> 3) & 15, j = 16 * I + (tid & 7), t = 16 * I + 8 + (r & 7);
    float s = 0.f;
#pragma unroll
    for (int kq = 0; kq < 4; ++kq) s += part[(kq * 4 + I) * 128 + r * 8 + (tid & 7)];
    if (r >= 8) Bm[t * LDA + j] = s;
    else if (DELTA) Am[t * LDA + j] = s * beta[t];
  }
#pragma unroll
  for (int u = 0; u < IT; ++u) {
    const int i = tid + u * 512, t = i / (DK / 4), d = (i % (DK / 4)) * 4;
    float4 q = *reinterpret_cast<float4*>(qf + t * LD + d), k = *reinterpret_cast<float4*>(kf + t * LD + d);
    const float4 l = *reinterpret_cast<float4*>(lf + t * LD + d), e = *reinterpret_cast<float4*>(tot + (t >> 4) * DK + d);
    *reinterpret_cast<float4*>(lf + t * LD + d) = make_float4(k.x * __expf(e.x - l.x), k.y * __expf(e.y - l.y), k.z * __expf(e.z - l.z), k.w * __expf(e.w - l.w));
    const float ex = __expf(l.x), ey = __expf(l.y), ez = __expf(l.z), ew = __expf(l.w);
    *reinterpret_cast<float4*>(qf + t * LD + d) = make_float4(q.x * ex, q.y * ey, q.z * ez, q.w * ew);
    *reinterpret_cast<float4*>(kf + t * LD + d) = make_float4(k.x * ex, k.y * ey, k.z * ez, k.w * ew);
  }
  if (tid < DK) {
    const float t0 = tot[tid], t1 = tot[DK + tid], t2 = tot[2 * DK + tid], t3 = tot[3 * DK + tid];
    const float f[10] = {t0, t0 + t1, t0 + t1 + t2, t0 + t1 + t2 + t3, t1 + t2 + t3, t2 + t3, t3, t1, t1 + t2, t2};
#pragma unroll
    for (int m = 0; m < 10; ++m) fac[m * DK + tid] = __expf(f[m]);
  }
  __syncthreads();
  // ---- A and B between blocks of 16: warps 0 - 5 queries of block I against keys of block J < I, 6 - 11 keys likewise (delta)
  if (warp < (DELTA ? 12 : 6)) {
    const int pr = warp % 6, I = pr < 1 ? 1 : pr < 3 ? 2 : 3, J = pr < 1 ? 0 : pr < 3 ? pr - 1 : pr - 3;
    const float* x = warp < 6 ? qf : kf;
    const float* f = I - J == 1 ? nullptr : fac + (J == 1 ? 9 : I == 2 ? 7 : 8) * DK;  // the blocks between them
    const int ta = 16 * I + g;
    float acc[2][4] = {};
#pragma unroll 4
    for (int k0 = 0; k0 < DK; k0 += 16) {
      uint32_t ah[4], al[4];
      uint4 bb[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int d = k0 + q2 + 8 * s;
        const float2 va = *reinterpret_cast<const float2*>(x + ta * LD + d), vb = *reinterpret_cast<const float2*>(x + (ta + 8) * LD + d);
        split2(va.x, va.y, ah[2 * s], al[2 * s]);
        split2(vb.x, vb.y, ah[2 * s + 1], al[2 * s + 1]);
        const float2 fd = f ? *reinterpret_cast<const float2*>(f + d) : make_float2(1.f, 1.f);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float2 kv = *reinterpret_cast<const float2*>(lf + (16 * J + nt * 8 + g) * LD + d);
          uint32_t hi, lo;
          split2(kv.x * fd.x, kv.y * fd.y, hi, lo);
          if (s) { bb[nt].y = hi; bb[nt].w = lo; } else { bb[nt].x = hi; bb[nt].z = lo; }
        }
      }
      mma3(acc[0], ah, al, bb[0]);
      mma3(acc[1], ah, al, bb[1]);
    }
    float* out = warp < 6 ? Bm : Am;
    const float fa = warp < 6 ? 1.f : beta[ta], fb = warp < 6 ? 1.f : beta[ta + 8];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int j = 16 * J + nt * 8 + q2;
      *reinterpret_cast<float2*>(out + ta * LDA + j) = make_float2(acc[nt][0] * fa, acc[nt][1] * fa);
      *reinterpret_cast<float2*>(out + (ta + 8) * LDA + j) = make_float2(acc[nt][2] * fb, acc[nt][3] * fb);
    }
  }
  __syncthreads();
  // ---- operands of the chain kernel; with the delta rule two warps invert the diagonal blocks of T = (I + Am)^-1 meanwhile, a column
  // per thread
  using Wk = Ws<DK>;
  uint4* ws = reinterpret_cast<uint4*>(a.ws) + ((size_t)(b * a.H + h) * gridDim.x + blockIdx.x) * Wk::total(a.DV, DELTA);
  constexpr int T0 = DELTA ? CT : 0, TN = 512 - T0;
  if (tid < T0) {
    const int blk = tid >> 4, cc = tid & 15;
    const float* Ld = Am + (blk * 16) * LDA + blk * 16;
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      float s = 0.f;
#pragma unroll
      for (int m = 0; m < r; ++m) s = fmaf(Ld[r * LDA + m], x[m], s);
      x[r] = r == cc ? 1.f : r < cc ? 0.f : -s;
      Tm[(blk * 16 + r) * LDA + blk * 16 + cc] = x[r];
    }
  } else {
    for (int i = tid - T0; i < Wk::Q; i += TN) {         // decayed queries: (token, channel pair)
      const int l = i & 31, ks = (i >> 5) % (DK / 16), nt = (i >> 5) / (DK / 16), t = nt * 8 + (l >> 2), d = ks * 16 + (l & 3) * 2, blk = t >> 4;
      float2 x = *reinterpret_cast<const float2*>(qf + t * LD + d), y = *reinterpret_cast<const float2*>(qf + t * LD + d + 8);
      if (blk) {
        const float2 f = *reinterpret_cast<const float2*>(fac + (blk - 1) * DK + d), f8 = *reinterpret_cast<const float2*>(fac + (blk - 1) * DK + d + 8);
        x.x *= f.x; x.y *= f.y; y.x *= f8.x; y.y *= f8.y;
      }
      uint4 o;
      split2(x.x, x.y, o.x, o.z);
      split2(y.x, y.y, o.y, o.w);
      ws[Wk::oQ + i] = o;
    }
    for (int i = tid - T0; i < Wk::K; i += TN) {         // decayed keys: (channel, token pair)
      const int l = i & 31, ks = (i >> 5) & 3, nt = i >> 7, d = nt * 8 + (l >> 2), t = ks * 16 + (l & 3) * 2;
      const float f = ks < 3 ? fac[(4 + ks) * DK + d] : 1.f;  // from the end of the block to the end of the chunk
      const float* p = lf + t * LD + d;
      uint4 o;
      split2(p[0] * f, p[LD] * f, o.x, o.z);
      split2(p[8 * LD] * f, p[9 * LD] * f, o.y, o.w);
      ws[Wk::oK + i] = o;
    }
    for (int i = tid - T0; i < Wk::B; i += TN) {
      const int l = i & 31, ks = (i >> 5) & 3, nt = i >> 7;
      const float* p = Bm + (nt * 8 + (l >> 2)) * LDA + ks * 16 + (l & 3) * 2;
      uint4 o;
      split2(p[0], p[1], o.x, o.z);
      split2(p[8], p[9], o.y, o.w);
      ws[Wk::oB + i] = o;
    }
    for (int d = tid - T0; d < DK; d += TN) reinterpret_cast<float*>(ws + Wk::oE)[d] = fac[3 * DK + d];
  }
  if constexpr (DELTA) {
    // ---- T by distance from the diagonal
    __syncthreads();
#pragma unroll 1
    for (int dist = 1; dist < 4; ++dist) {
      const int items = (4 - dist) * 256;
      for (int i = tid; i < items; i += 512) {           // sum_m L_Im T_mJ
        const int J = i >> 8, I = J + dist, r = (i >> 4) & 15, cc = i & 15;
        float s = 0.f;
        for (int m0 = J * 16; m0 < I * 16; m0 += 16)
#pragma unroll
          for (int m = m0; m < m0 + 16; ++m) s = fmaf(Am[(I * 16 + r) * LDA + m], Tm[m * LDA + J * 16 + cc], s);
        tmp[J * 272 + r * 17 + cc] = s;
      }
      __syncthreads();
      for (int i = tid; i < items; i += 512) {
        const int J = i >> 8, I = J + dist, r = (i >> 4) & 15, cc = i & 15;
        float s = 0.f;
#pragma unroll
        for (int m = 0; m < 16; ++m) s = fmaf(Tm[(I * 16 + r) * LDA + I * 16 + m], tmp[J * 272 + m * 17 + cc], s);
        Tm[(I * 16 + r) * LDA + J * 16 + cc] = -s;
      }
      __syncthreads();
    }
    // ---- W and U': 16 columns of [K e^c | V] per warp and turn
    const int n_w = DK / 16, n_all = n_w + a.DV / 16;
    float* up = reinterpret_cast<float*>(ws + Wk::oU);
    for (int ct = warp; ct < n_all; ct += 16) {
      const bool is_w = ct < n_w;
      const int col0 = is_w ? ct * 16 : (ct - n_w) * 16;
      float v[4][2][4];                                  // all loads in flight
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const int col = col0 + nt * 8 + g;
          const float f = is_w && ks ? fac[(ks - 1) * DK + col] : 1.f;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int t = ks * 16 + q2 + (u & 1) + (u >> 1) * 8;
            v[ks][nt][u] = is_w ? kf[t * LD + col] * f : a.v[(row0 + min(t, n - 1)) * a.ld_v + (size_t)h * a.DV + col];
          }
        }
      float acc[4][2][4] = {};
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint4 bb[2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int t = ks * 16 + q2 + (u & 1) + (u >> 1) * 8;
            v[ks][nt][u] = t < n ? beta[t] * v[ks][nt][u] : 0.f;
          }
          split2(v[ks][nt][0], v[ks][nt][1], bb[nt].x, bb[nt].z);
          split2(v[ks][nt][2], v[ks][nt][3], bb[nt].y, bb[nt].w);
        }
#pragma unroll
        for (int mt = ks; mt < 4; ++mt) {
          uint32_t ah[4], al[4];
          const float* p = Tm + (mt * 16 + g) * LDA + ks * 16 + q2;
          const float2 t0 = *reinterpret_cast<const float2*>(p), t1 = *reinterpret_cast<const float2*>(p + 8 * LDA);
          const float2 t2 = *reinterpret_cast<const float2*>(p + 8), t3 = *reinterpret_cast<const float2*>(p + 8 * LDA + 8);
          split2(t0.x, t0.y, ah[0], al[0]); split2(t1.x, t1.y, ah[1], al[1]);
          split2(t2.x, t2.y, ah[2], al[2]); split2(t3.x, t3.y, ah[3], al[3]);
          mma3(acc[mt][0], ah, al, bb[0]);
          mma3(acc[mt][1], ah, al, bb[1]);
        }
      }
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int u = 0; u < 2; ++u) {                    // tokens mt * 16 + g (+ 8): token tile 2 mt + u
          if (is_w) {                                    // accumulator and operand layouts agree lane by lane
            uint4 o;
            split2(acc[mt][0][2 * u], acc[mt][0][2 * u + 1], o.x, o.z);
            split2(acc[mt][1][2 * u], acc[mt][1][2 * u + 1], o.y, o.w);
            ws[((2 * mt + u) * n_w + ct) * 32 + lane] = o;
          } else {
            float* p = up + (size_t)(mt * 16 + u * 8 + g) * a.DV + col0 + q2;
            *reinterpret_cast<float2*>(p) = make_float2(acc[mt][0][2 * u], acc[mt][0][2 * u + 1]);
            *reinterpret_cast<float2*>(p + 8) = make_float2(acc[mt][1][2 * u], acc[mt][1][2 * u + 1]);
          }
        }
    }
  }
}

// ---------------------------------------------------------------------------------------------- 2. the chain over the chunks
// grid (DV / 16, H, B); DK / 16 warps, warp w owns key channels 16 w .. 16 w + 15 of S^T and the token tiles w, w + DK / 16, ..
// Bound by shared memory's and L1's throughput (65 % with the waits around its two barriers) and by latencies.  The operand blocks, of
// which every one is read once, come straight into registers, asked for where the block of the chunk before was used last; through shared
// memory (written and read: half of its traffic) it took two more barriers a chunk: 2048 tokens, 16 heads of 128 x 128 89.6 -> 78 us, 3 x 701 tokens,
// 8 heads of 128 x 256 without the delta rule 67.6 -> 56.  The state shared as an operand in place of the partial products' exchange:
// 76 -> 71 us alone, nothing for a prompt, and 56 -> 60.
template <int DK, bool DELTA>
__global__ void __launch_bounds__(DK * 2, 1) channel_chain_kernel(RecurArgs a, int c0, int NC) {
  extern __shared__ __align__(16) uint4 sm4[];
  using Wk = Ws<DK>;
  constexpr int NW = DK / 16, TH = DK * 2, TPW = 8 / NW;
  float4* exU = reinterpret_cast<float4*>(sm4);          // [warp][token tile][lane] partial products with S
  float4* exO = exU + (DELTA ? NW * 256 : 0);
  uint4* sU = reinterpret_cast<uint4*>(exO + NW * 256);  // U^T as left operand: [k step 4][hi, lo][lane]
  pdl_launch();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q2 = (lane & 3) * 2;
  const int e0 = blockIdx.x * 16, h = blockIdx.y, b = blockIdx.z;
  const size_t per = Wk::total(a.DV, DELTA);
  const uint4* ws = reinterpret_cast<const uint4*>(a.ws) + (size_t)(b * a.H + h) * NC * per;
  const int O = a.H * a.DV;
  float* st = a.state + ((size_t)b * a.H + h) * DK * a.DV + e0;
  float sacc[2][4];                                      // S^T: value column g (+ 8), channel 16 warp + 8 t + q2 (+ 1)
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int u = 0; u < 4; ++u) sacc[t][u] = st[(size_t)(warp * 16 + t * 8 + q2 + (u & 1)) * a.DV + g + (u >> 1) * 8];
  // Operands of the chunk at hand; each is asked for anew for the next chunk where it was used last
  uint4 rW[DELTA ? 8 : 1], rQ[8], rK[2][4], rB[TPW][4];
  float uv[TPW][4], ec[2][2];  // U' or V at value columns g, g + 8 and tokens q2, q2 + 1 of this lane's tiles; the chunk's decays
  auto get_q = [&](int c, int nt) {
    const uint4* w = ws + (size_t)c * per + (nt * NW + warp) * 32 + lane;
    if (DELTA) rW[nt] = __ldcg(w);
    rQ[nt] = __ldcg(w + Wk::oQ);
  };
  auto get_k = [&](int c, int ks) {
    const uint4* w = ws + (size_t)c * per + ks * 32 + lane;
#pragma unroll
    for (int t = 0; t < 2; ++t) rK[t][ks] = __ldcg(w + Wk::oK + (warp * 2 + t) * 128);
#pragma unroll
    for (int p = 0; p < TPW; ++p)
      if (ks <= (warp + p * NW) >> 1) rB[p][ks] = __ldcg(w + Wk::oB + (warp + p * NW) * 128);  // keys up to the query
  };
  auto get_u = [&](int c, int p) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = (warp + p * NW) * 8 + q2 + (u & 1), e = e0 + g + (u >> 1) * 8;
      if (DELTA) uv[p][u] = __ldcg(reinterpret_cast<const float*>(ws + (size_t)c * per + Wk::oU) + (size_t)t * a.DV + e);
      else uv[p][u] = (c0 + c) * CT + t < a.L ? a.v[((size_t)b * a.L + (size_t)(c0 + c) * CT + t) * a.ld_v + (size_t)h * a.DV + e] : 0.f;
    }
  };
  auto get_e = [&](int c) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const float2 v = __ldcg(reinterpret_cast<const float2*>(reinterpret_cast<const float*>(ws + (size_t)c * per + Wk::oE) + warp * 16 + t * 8 + q2));
      ec[t][0] = v.x; ec[t][1] = v.y;
    }
  };
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) get_q(0, nt);
#pragma unroll
  for (int p = 0; p < TPW; ++p) get_u(0, p);
  get_e(0);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) get_k(0, ks);
#pragma unroll 1
  for (int c = 0; c < NC; ++c) {
    const int n = min(CT, a.L - (c0 + c) * CT);
    const size_t row0 = (size_t)b * a.L + (size_t)(c0 + c) * CT;
    const bool more = c + 1 < NC;
    {
      uint32_t ah[4], al[4];
      split2(sacc[0][0], sacc[0][1], ah[0], al[0]); split2(sacc[0][2], sacc[0][3], ah[1], al[1]);
      split2(sacc[1][0], sacc[1][1], ah[2], al[2]); split2(sacc[1][2], sacc[1][3], ah[3], al[3]);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        if (DELTA) {
          float p[4] = {};
          mma3(p, ah, al, rW[nt]);
          exU[(warp * 8 + nt) * 32 + lane] = make_float4(p[0], p[1], p[2], p[3]);
        }
        float p[4] = {};
        mma3(p, ah, al, rQ[nt]);
        exO[(warp * 8 + nt) * 32 + lane] = make_float4(p[0], p[1], p[2], p[3]);
        if (more) get_q(c + 1, nt);
      }
    }
    __syncthreads();
    float o[TPW][4];
#pragma unroll
    for (int p = 0; p < TPW; ++p) {
      const int nt = warp + p * NW;
      float4 so = make_float4(0.f, 0.f, 0.f, 0.f), su = so;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const float4 x = exO[(w * 8 + nt) * 32 + lane];
        so.x += x.x; so.y += x.y; so.z += x.z; so.w += x.w;
        if (DELTA) {
          const float4 y = exU[(w * 8 + nt) * 32 + lane];
          su.x += y.x; su.y += y.y; su.z += y.z; su.w += y.w;
        }
      }
      o[p][0] = so.x; o[p][1] = so.y; o[p][2] = so.z; o[p][3] = so.w;
      float u0 = uv[p][0], u1 = uv[p][1], u2 = uv[p][2], u3 = uv[p][3];
      if (DELTA) { u0 -= su.x; u1 -= su.y; u2 -= su.z; u3 -= su.w; }
      if (more) get_u(c + 1, p);
      uint2 hi, lo;                                      // half of an operand's four registers: tokens (nt & 1) * 8 + q2 of step nt / 2
      split2(u0, u1, hi.x, lo.x);
      split2(u2, u3, hi.y, lo.y);
      uint2* dst = reinterpret_cast<uint2*>(sU + ((nt >> 1) * 2) * 32 + lane) + (nt & 1);
      dst[0] = hi;
      dst[64] = lo;                                      // 32 lanes of 16 bytes further
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 2; ++t) { sacc[t][0] *= ec[t][0]; sacc[t][1] *= ec[t][1]; sacc[t][2] *= ec[t][0]; sacc[t][3] *= ec[t][1]; }
    if (more) get_e(c + 1);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const uint4 uh = sU[(ks * 2) * 32 + lane], ul = sU[(ks * 2 + 1) * 32 + lane];
      const uint32_t ah[4] = {uh.x, uh.y, uh.z, uh.w}, al[4] = {ul.x, ul.y, ul.z, ul.w};
#pragma unroll
      for (int t = 0; t < 2; ++t) mma3(sacc[t], ah, al, rK[t][ks]);
#pragma unroll
      for (int p = 0; p < TPW; ++p)
        if (ks <= (warp + p * NW) >> 1) mma3(o[p], ah, al, rB[p][ks]);
      if (more) get_k(c + 1, ks);
    }
#pragma unroll
    for (int p = 0; p < TPW; ++p)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = (warp + p * NW) * 8 + q2 + (u & 1);
        if (t < n) a.out[(row0 + t) * O + (size_t)h * a.DV + e0 + g + (u >> 1) * 8] = o[p][u];
      }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int u = 0; u < 4; ++u) st[(size_t)(warp * 16 + t * 8 + q2 + (u & 1)) * a.DV + g + (u >> 1) * 8] = sacc[t][u];
}

template <int DK> size_t per_chunk(int DV, bool delta) { return Ws<DK>::total(DV, delta) * 4; }  // floats

template <int DK, bool DELTA>
cudaError_t launch_channel_t(const RecurArgs& a, cudaStream_t s) {
  using Wk = Ws<DK>;
  const size_t sm1 = (size_t)chunk_floats<DK>(DELTA) * sizeof(float);
  const size_t sm2 = (size_t)((DELTA ? 2 : 1) * (DK / 16) * 256 + 256) * 16;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(channel_chunk_kernel<DK, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(channel_chain_kernel<DK, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2)) != cudaSuccess) return e;
  const int NC = (a.L + CT - 1) / CT;
  const int seg = (int)std::min<size_t>(NC, a.ws_floats / ((size_t)a.B * a.H * per_chunk<DK>(a.DV, DELTA)));  // chunks the workspace holds
  for (int c0 = 0; c0 < NC; c0 += seg) {
    const int nc = std::min(seg, NC - c0);
    if ((e = launch_k(channel_chunk_kernel<DK, DELTA>, dim3(nc, a.H, a.B), dim3(512), sm1, s, a, c0)) != cudaSuccess) return e;
    if ((e = launch_k(channel_chain_kernel<DK, DELTA>, dim3(a.DV / 16, a.H, a.B), dim3(DK * 2), sm2, s, a, c0, nc)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

bool recur_channel_shape(int DK, int DV) { return (DK == 64 || DK == 128) && DV % 16 == 0 && DV >= 16; }

size_t recur_channel_ws_floats(int B, int L, int H, int DK, int DV) {
  const size_t per = DK == 64 ? per_chunk<64>(DV, true) : per_chunk<128>(DV, true);
  return (size_t)B * H * ((L + CT - 1) / CT) * per;
}

// Portions from this length on.  A chunk's CTA takes ~13 us (gated linear attention: 264 of them in 26 us) to ~21 us (delta rule, with the
// triangular system: 512 in 86 us, one per SM at a time) whatever it holds; the chain takes 0.2 - 0.3 us per token, and more where its
// CTAs (a multiple of sequences x heads) fill the chip.  One layer, prompt through the public call, chain : chunks in us: delta rule, 1 x
// 16 heads, 48 tokens 248 : 258, 64 258 : 262, 96 283 : 281, 128 306 : 293, 192 278 : 254, 400 360 : 278; 1 x 4 heads, 64 219 : 223, 96
// 239 : 238, 128 261 : 249; 4 x 16 heads, 32 401 : 438, 48 359 : 359, 64 376 : 367, 128 445 : 395.  Gated linear attention, 1 x 2 heads,
// 32 152 : 154, 48 166 : 165, 64 174 : 166, 72 186 : 176, 128 215 : 189 (it would not lose from 48 on; the line is from when a chunk took
// longer); 1 x 8 heads, 48 212 : 203, 64 218 : 203, 128 254 : 221; 4 x 8 heads, 32 341 : 348, 48 349 : 335.
static int least_tokens(const RecurArgs& a) {
  if (a.mode == 1) return a.B * a.H >= 64 ? 64 : 128;
  return a.B * a.H >= 8 ? RECUR_CHANNEL_MIN : 72;
}

bool recur_channel_supported(const RecurArgs& a) {
  static const bool on = !(getenv("L3_RECUR_CHUNK") && atoi(getenv("L3_RECUR_CHUNK")) == 0);
  if (!on || !a.bf16_ops || !a.ws || a.L < least_tokens(a) || !recur_channel_shape(a.DK, a.DV)) return false;
  if ((a.mode != 1 && a.mode != 2) || !a.log_c || a.act_in || a.q_mul != 0.f || a.n_state || a.k_scale) return false;
  const uintptr_t al = (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.log_c | (uintptr_t)a.ws;
  if (a.ld_q % 4 || a.ld_k % 4 || (al & 15)) return false;
  return recur_channel_ws_floats(a.B, 1, a.H, a.DK, a.DV) <= a.ws_floats;
}

cudaError_t launch_recur_channel(const RecurArgs& a, cudaStream_t s) {
  if (!recur_channel_supported(a)) return cudaErrorInvalidValue;
  if (a.DK == 64) return a.mode == 1 ? launch_channel_t<64, true>(a, s) : launch_channel_t<64, false>(a, s);
  return a.mode == 1 ? launch_channel_t<128, true>(a, s) : launch_channel_t<128, false>(a, s);
}
