// Prompt attention in fp32 (llama3.py:190-211 for L > 1; windows, kept tokens, sinks, sigmoid weights and output gates of the layer lists):
// fp32 queries, keys, values, weights and sums, FFMA throughout.
//
// A CTA holds 32 query rows of one key head - row = (token, query head of the group), token-major - and walks the keys they can see, 64 at
// a time.  Warp w owns the rows 8 (w & 3) .. + 7 over the keys 32 (w >> 2) .. + 31 of every tile with a softmax state of its own, so that
// nothing but a tile's arrival is waited for by all; the parts of the keys meet once at the end.  Two groups of 8 warps take every second
// tile each where a launch is one CTA per SM, whether by its grid or by its shared memory: one loads while the other multiplies, and the
// longest row of tiles is half as long.  Where two CTAs share an SM they do that for one another.
//   scores   a lane has 2 rows x 4 keys and reads 16-byte pieces along the head: 6 shared-memory wavefronts (rows padded to an odd number
//            of pieces: no conflicts) feed 16 pairs of products per lane, summed as even and odd entries
//   output   a lane has 4 rows x 4 NC value columns; the weights arrive through shared memory, a warp's own, as broadcasts
// What bounds it: the FFMA pipe (a tile of 32 x 64 with heads of 192 | 128 is 655 k products, 128 a cycle), then the latency of a tile.  The
// kernels it took over from read 12 wavefronts per 8 cycles of products and loaded each tile in between (attn_window.cu), or had a barrier
// between scores, softmax and output (attention.cu).  600 tokens, 8 heads of 192 | 128: 123.5 -> 79 us a layer.
// A warp's output loop runs over the keys that one of its eight rows sees: values of other keys - a NaN or an infinity in a later token -
// do not reach it.
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"
#include "mixer.h"
#include "../../include/llama3_b200.h"

namespace {

constexpr int FR = 32, FK = 64, FW = 8;  // query rows, keys per tile, warps

__host__ __device__ inline int row_ld(int dk) { return dk / 4 % 2 ? dk : dk + 4; }
__host__ __device__ inline int stage_floats(int dk, int dv) { return FK * (row_ld(dk) + dv); }
size_t smem_bytes(int dk, int dv, int gr) {
  return ((size_t)FR * row_ld(dk) + (size_t)gr * (stage_floats(dk, dv) + FW * 32 * 8)) * sizeof(float);
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool in) {  // zeros where there is no such key
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }

// NC: pieces of 64 value columns; GR: groups of 8 warps, each with every GR-th tile of keys
template <int NC, int GR>
__global__ void __launch_bounds__(32 * FW * GR, GR == 1 && NC <= 2 ? 2 : 1) attn_f32_kernel(WinAttnArgs a) {
  extern __shared__ __align__(16) float sm[];
  const int DK = a.DK, DV = a.DV, KS = row_ld(DK), ST = stage_floats(DK, DV);
  float* sQ = sm;                        // [32][KS]
  float* sT = sQ + FR * KS;              // [groups][64 keys of KS | 64 values of DV]
  float* sP = sT + GR * ST;              // [warps][32 keys][8 rows]
  pdl_launch();
  pdl_wait();
  const int group = GR == 1 ? 0 : threadIdx.x / (32 * FW), tid = threadIdx.x - group * 32 * FW, lane = tid & 31, warp = tid >> 5;  // in the group
  const int rep = a.H / a.G, g = blockIdx.y, b = blockIdx.z;
  const int nrows = a.L * rep;
  const int row0 = (gridDim.x - 1 - blockIdx.x) * FR;  // late tokens see the most keys: their tiles start first
  const int pos0 = *a.pos_ptr;
  const int p_lo = pos0 + row0 / rep, p_hi = pos0 + min(a.L - 1, (row0 + FR - 1) / rep);
  auto first_key = [&](int p) { return a.window <= 0 ? 0 : a.chunked ? p - p % a.window : max(0, p - a.window + 1); };
  // keys the tile can see: [0, ka) kept tokens ahead of the window, then [w_lo, p_hi]
  const int w_lo = first_key(p_lo), ka = min(a.keep_first, w_lo), nkeys = ka + (p_hi + 1 - w_lo);
  const int ntiles = (nkeys + FK - 1) / FK;
  const int dk1 = DK - a.dk2, k_ld = a.k_ld ? a.k_ld : DK, v_ld = a.k_ld ? a.k_ld : DV;
  const float* ck = (const float*)a.cache_k + (a.k_ld ? (size_t)b * a.kv_seq + (size_t)g * dk1 : ((size_t)b * a.G + g) * a.M * DK);
  const float* cv = (const float*)a.cache_v + (a.k_ld ? (size_t)b * a.kv_seq + (size_t)g * DV : ((size_t)b * a.G + g) * a.M * DV);
  const float* ck2 = (const float*)a.k2 + (size_t)b * a.k2_seq;

  float* st = sT + group * ST;
  auto load = [&](int tile) {  // 8 threads per key
    for (int kk = tid >> 3; kk < FK; kk += 32 * FW / 8) {
      const int vi = tile * FK + kk;
      const bool in = vi < nkeys;
      const size_t j = in ? (vi < ka ? vi : w_lo + (vi - ka)) : 0;
      float *dk = st + kk * KS, *dv = st + FK * KS + kk * DV;
      for (int c = 4 * (tid & 7); c < dk1; c += 32) cp16(dk + c, ck + j * k_ld + c, in);
      for (int c = 4 * (tid & 7); c < a.dk2; c += 32) cp16(dk + dk1 + c, ck2 + j * a.k2_ld + c, in);
      for (int c = 4 * (tid & 7); c < DV; c += 32) cp16(dv + c, cv + j * v_ld + c, in);
    }
  };
  auto group_sync = [&]() {
    if (GR == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(32 * FW) : "memory");
  };
  for (int rr = threadIdx.x >> 3; rr < FR; rr += 32 * FW * GR / 8) {
    const int row = row0 + rr, t = row < nrows ? row / rep : 0, h = g * rep + (row < nrows ? row - t * rep : 0);
    const float* src = a.q + (((size_t)b * a.L + t) * a.H + h) * DK;
    for (int c = 4 * (threadIdx.x & 7); c < DK; c += 32) cp16(sQ + rr * KS + c, src + c, row < nrows);
  }
  if (group < ntiles) load(group);
  cp_wait_all();
  __syncthreads();

  // scores: rows 2 rg + i of the warp's eight, keys kg + 8 j of its 32; output: rows 4 rp + r, columns 4 cg + 64 c
  const int rg = lane >> 3, kg = lane & 7, rp = lane >> 4, cg = lane & 15;
  const int wrow = row0 + 8 * (warp & 3), half = warp >> 2;
  const bool live = wrow < nrows;
  const int pw_lo = pos0 + wrow / rep, pw_hi = pos0 + min(wrow + 7, nrows - 1) / rep;  // positions of the warp's rows
  const int seen = ka + pw_hi + 1 - w_lo;                                             // keys from the tile's list that they see at most
  const int unseen = a.keep_first <= w_lo ? ka + first_key(pw_lo) - w_lo : 0;         // keys behind the kept ones that none of them sees any more
  float mx[2], sum[2], hv[2];
  int rpos[2], rlo[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int row = wrow + 2 * rg + i, t = row / rep;
    rpos[i] = row < nrows ? pos0 + t : -1;
    rlo[i] = row < nrows ? first_key(pos0 + t) : 0;
    hv[i] = a.head_vec ? a.head_vec[g * rep + row - t * rep] : 0.f;
    const bool sink = a.kind == L3_ATTN_SINK && a.head_vec && half == 0 && group == 0;
    mx[i] = sink ? hv[i] : -INFINITY;
    sum[i] = sink && kg == 0 ? 1.f : 0.f;  // summed over the lanes of a row at the end
  }
  float2 o[4][NC][2];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < NC; ++c) o[r][c][0] = o[r][c][1] = make_float2(0.f, 0.f);
  float* myP = sP + (group * FW + warp) * 32 * 8;
  auto of_row = [&](const float (&v)[2], int r) { return __shfl_sync(L3_FULL, v[r & 1], 8 * (2 * rp + (r >> 1))); };

  for (int tile = group; tile < ntiles; tile += GR) {
    if (tile > group) {
      group_sync();  // nobody reads the tile before this one any more
      load(tile);
      cp_wait_all();
      group_sync();
    }
    const int v0 = tile * FK + 32 * half;
    const int k_end = min(32, seen - v0), k_beg = v0 >= ka ? max(0, unseen - v0) : 0;
    if (live && k_beg < k_end) {
      const float* q = sQ + (8 * (warp & 3) + 2 * rg) * KS;
      const float* k = st + (32 * half + kg) * KS;
      float2 s2[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2[i][j] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int d = 0; d < DK; d += 4) {
        float4 qv[2], kv[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) qv[i] = *reinterpret_cast<const float4*>(q + i * KS + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(k + 8 * j * KS + d);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            s2[i][j] = fma2(make_float2(qv[i].x, qv[i].y), make_float2(kv[j].x, kv[j].y), s2[i][j]);
            s2[i][j] = fma2(make_float2(qv[i].z, qv[i].w), make_float2(kv[j].z, kv[j].w), s2[i][j]);
          }
      }
      float w[2][4], alpha[2] = {1.f, 1.f};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        bool vis[4];
        float top = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int vi = v0 + kg + 8 * j, key = vi < ka ? vi : w_lo + (vi - ka);
          vis[j] = vi < nkeys && key <= rpos[i] && (key >= rlo[i] || key < a.keep_first);
          w[i][j] = (s2[i][j].x + s2[i][j].y) * a.scale;
          if (vis[j]) top = fmaxf(top, w[i][j]);
        }
        if (a.kind == L3_ATTN_SIGMOID) {
#pragma unroll
          for (int j = 0; j < 4; ++j) w[i][j] = vis[j] ? sigmoid_f(w[i][j] + hv[i]) : 0.f;
        } else {
#pragma unroll
          for (int off = 1; off < 8; off <<= 1) top = fmaxf(top, __shfl_xor_sync(L3_FULL, top, off));
          const float m = fmaxf(mx[i], top);
          alpha[i] = m == -INFINITY ? 1.f : expf(mx[i] - m);
          mx[i] = m;
          sum[i] *= alpha[i];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            w[i][j] = vis[j] ? expf(w[i][j] - m) : 0.f;
            sum[i] += w[i][j];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(myP + (kg + 8 * j) * 8 + 2 * rg) = make_float2(w[0][j], w[1][j]);
      if (__any_sync(L3_FULL, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float f = of_row(alpha, r);
#pragma unroll
          for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) { o[r][c][e].x *= f; o[r][c][e].y *= f; }
        }
      }
      __syncwarp();
      const float* v = st + FK * KS + 32 * half * DV;
#pragma unroll 2
      for (int kk = k_beg; kk < k_end; ++kk) {
        const float4 p4 = *reinterpret_cast<const float4*>(myP + kk * 8 + 4 * rp);
        const float2 p[4] = {make_float2(p4.x, p4.x), make_float2(p4.y, p4.y), make_float2(p4.z, p4.z), make_float2(p4.w, p4.w)};
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int d = 4 * cg + 64 * c;
          const float4 x = *reinterpret_cast<const float4*>(v + kk * DV + (d < DV ? d : 0));
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            o[r][c][0] = fma2(p[r], make_float2(x.x, x.y), o[r][c][0]);
            o[r][c][1] = fma2(p[r], make_float2(x.z, x.w), o[r][c][1]);
          }
        }
      }
      __syncwarp();
    }
  }
  // the two halves of the keys
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int off = 1; off < 8; off <<= 1) sum[i] += __shfl_xor_sync(L3_FULL, sum[i], off);
  __syncthreads();
  const int src = 2 * group + half;  // states of the keys: 0 stays in registers
  float* sO = sT;                    // [parts - 1][32 rows][DV]: at most half of the stages
  float* sML = sP;                   // [parts - 1][32 rows] (max, sum)
  if (src > 0) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int rr = (src - 1) * FR + 8 * (warp & 3) + 4 * rp + r;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int d = 4 * cg + 64 * c;
        if (d < DV) *reinterpret_cast<float4*>(sO + rr * DV + d) = make_float4(o[r][c][0].x, o[r][c][0].y, o[r][c][1].x, o[r][c][1].y);
      }
    }
    if (kg == 0)
#pragma unroll
      for (int i = 0; i < 2; ++i) *reinterpret_cast<float2*>(sML + 2 * ((src - 1) * FR + 8 * (warp & 3) + 2 * rg + i)) = make_float2(mx[i], sum[i]);
  }
  __syncthreads();
  if (src > 0 || !live) return;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int rr = 8 * (warp & 3) + 4 * rp + r, row = row0 + rr;
    const float m0 = of_row(mx, r), l0 = of_row(sum, r);
    if (row >= nrows) continue;
    float f[2 * GR], mul = a.out_scale;
    f[0] = 1.f;
#pragma unroll
    for (int i = 1; i < 2 * GR; ++i) f[i] = 1.f;
    if (a.kind != L3_ATTN_SIGMOID) {
      float2 ml[2 * GR];
      ml[0] = make_float2(m0, l0);
      float m = m0;
#pragma unroll
      for (int i = 1; i < 2 * GR; ++i) {
        ml[i] = *reinterpret_cast<const float2*>(sML + 2 * ((i - 1) * FR + rr));
        m = fmaxf(m, ml[i].x);
      }
      float l = 0.f;
#pragma unroll
      for (int i = 0; i < 2 * GR; ++i) {
        f[i] = ml[i].x == -INFINITY ? 0.f : expf(ml[i].x - m);
        l += ml[i].y * f[i];
      }
      mul *= l > 0.f ? 1.0f / l : 0.f;
    }
    const int t = row / rep, h = g * rep + row - t * rep;
    const size_t gr = (size_t)b * a.L + t;
    if (a.gate && !a.gate_wide) mul *= sigmoid_f(a.gate[gr * a.ld_gate + h]);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int d = 4 * cg + 64 * c;
      if (d >= DV) continue;
      float v[4] = {o[r][c][0].x * f[0], o[r][c][0].y * f[0], o[r][c][1].x * f[0], o[r][c][1].y * f[0]};
#pragma unroll
      for (int i = 1; i < 2 * GR; ++i) {
        const float4 y = *reinterpret_cast<const float4*>(sO + ((i - 1) * FR + rr) * DV + d);
        v[0] += y.x * f[i]; v[1] += y.y * f[i]; v[2] += y.z * f[i]; v[3] += y.w * f[i];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[e] *= mul;
        if (a.gate && a.gate_wide) v[e] *= sigmoid_f(a.gate[gr * a.ld_gate + (size_t)h * DV + d + e]);
      }
      const size_t oi = gr * a.ld_out + (size_t)h * DV + d;
      if (a.out_lo) {
        float4 hi, lo;
        split_tf32(v[0], hi.x, lo.x); split_tf32(v[1], hi.y, lo.y); split_tf32(v[2], hi.z, lo.z); split_tf32(v[3], hi.w, lo.w);
        *reinterpret_cast<float4*>(a.out + oi) = hi;
        *reinterpret_cast<float4*>(a.out_lo + oi) = lo;
      } else if (a.out) *reinterpret_cast<float4*>(a.out + oi) = make_float4(v[0], v[1], v[2], v[3]);
      if (a.out16) {
        union { __nv_bfloat162 h2[2]; uint2 u; } pk;
        pk.h2[0] = __floats2bfloat162_rn(v[0], v[1]);
        pk.h2[1] = __floats2bfloat162_rn(v[2], v[3]);
        *reinterpret_cast<uint2*>(a.out16 + oi) = pk.u;
      }
    }
  }
}

template <int NC, int GR> cudaError_t launch_gr(const WinAttnArgs& a, dim3 grid, cudaStream_t s) {
  const size_t smem = smem_bytes(a.DK, a.DV, GR);
  if (const cudaError_t e = allow_smem(attn_f32_kernel<NC, GR>, smem)) return e;
  return launch_k(attn_f32_kernel<NC, GR>, grid, dim3(32 * FW * GR), smem, s, a);
}
template <int NC> cudaError_t launch_nc(const WinAttnArgs& a, cudaStream_t s) {
  const dim3 grid((a.L * (a.H / a.G) + FR - 1) / FR, a.G, a.B);
  const long ctas = (long)grid.x * grid.y * grid.z;
  // One CTA per SM: two groups, us with one : two.  Grids of up to one CTA per SM, vupitar width 512, 800 tokens 784 : 712; up to two, debuzen
  // width 1024, 800 tokens 2230 : 2146; above, and with one tile of keys to walk, within 1 %.  (296: twice the SMs.  The instance of 256 value
  // columns and two groups spills 136 bytes; over value sizes of 160 - 256, 40 - 800 tokens, it takes 0.88 - 1.01 of the tiled kernel's time.)
  const bool fits = smem_bytes(a.DK, a.DV, 2) <= 220 * 1024, pair = smem_bytes(a.DK, a.DV, 1) <= 113 * 1024;
  return fits && (!pair || (a.L > FK && ctas <= 296)) ? launch_gr<NC, 2>(a, grid, s) : launch_gr<NC, 1>(a, grid, s);
}

}  // namespace

// every row of q, keys, values and outputs in whole 16-byte pieces
bool attn_f32_supported(const WinAttnArgs& a) {
  const uintptr_t p = (uintptr_t)a.q | (uintptr_t)a.cache_k | (uintptr_t)a.cache_v | (uintptr_t)a.k2 | (uintptr_t)a.out | (uintptr_t)a.out_lo | (uintptr_t)a.out16;
  return a.nsplit == 1 && a.L > 1 && a.DK % 4 == 0 && a.DV % 4 == 0 && a.dk2 % 4 == 0 && a.k_ld % 4 == 0 && a.k2_ld % 4 == 0 && a.kv_seq % 4 == 0 &&
         a.k2_seq % 4 == 0 && a.ld_out % 4 == 0 && p % 16 == 0 && a.DV <= 256 && smem_bytes(a.DK, a.DV, 1) <= 220 * 1024;
}

cudaError_t launch_attn_f32(const WinAttnArgs& a, cudaStream_t s) {
  if (!attn_f32_supported(a)) return cudaErrorInvalidValue;
  return a.DV <= 64 ? launch_nc<1>(a, s) : a.DV <= 128 ? launch_nc<2>(a, s) : launch_nc<4>(a, s);
}
