// Row kernels around the token mixers of layer-list decoders (layerlist.cu): everything here is fp32 - norms,
// gates, the residual sum - whatever the model's weight type is.
//
//  * resid_postnorm_kernel   x += mult * y / rms(y) * w        (norm on the sublayer's OUTPUT), emits the bf16
//                            mirror of the new residual row for the tensor-core projections that read it next
//  * gated_rmsnorm_kernel    out = o / rms_group(o) * w * sigmoid(gate)   over the whole row or per head
//  * qk_norm_cache_kernel    RMS norm over the WHOLE q / k projection, append k (normalised) and the raw k
//                            (the values of this attention) to the KV cache
//  * side_mul_kernel         act(g) * E[token, layer slice]    (per-layer token input)
//  * delta_prep_kernel       short causal convolutions + silu, unit-length q / k, decay and write strength of
//                            the gated delta rule; conv_tail_kernel moves the convolutions' tails on (a call of one
//                            token lets delta_prep_kernel do that itself)
//  * rmsnorm_rows_kernel     plain RMS norm of chosen rows, any width (ahead of the LM head)
//  * to_bf16_kernel          bf16 mirror of fp32 rows
#include <algorithm>

#include "common.cuh"
#include "mixer.h"
#include "rowvec.cuh"

namespace {

__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

// sum over the CTA (every thread gets the total; same order of additions in every thread)
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();  // red may still be read from a previous call
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < nw; ++w) t += red[w];
  return t;
}

__global__ void __launch_bounds__(256) resid_postnorm_kernel(float* __restrict__ x, const float* __restrict__ y,
                                                             const float* __restrict__ w, float mult, float eps, int D,
                                                             bf16* __restrict__ x16) {
  __shared__ float red[32];
  pdl_launch();
  pdl_wait();
  const size_t r = blockIdx.x;
  const float* yr = y + r * D;
  float ss = 0.f;
  for (int i = threadIdx.x; i < D; i += blockDim.x) { const float v = yr[i]; ss = fmaf(v, v, ss); }
  const float rinv = 1.0f / sqrtf(block_sum(ss, red) / (float)D + eps);
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const float v = x[r * D + i] + mult * (yr[i] * rinv * w[i]);
    x[r * D + i] = v;
    if (x16) x16[r * D + i] = __float2bfloat16_rn(v);
  }
}

// the same over rows in registers.  2048 x 2048: 19.8 -> 10.0 us
template <int NV>
__global__ void __launch_bounds__(256) resid_postnorm_vec_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ w,
                                                                 float mult, float eps, int D, bf16* __restrict__ x16) {
  __shared__ float red[32];
  pdl_launch();
  pdl_wait();
  const size_t r = blockIdx.x;
  float4 yv[NV], xv[NV], wv[NV];
  row_load(y + r * D, D, yv);
  row_load(x + r * D, D, xv);
  row_load(w, D, wv);
  float ss = 0.f;
#pragma unroll
  for (int u = 0; u < NV; ++u) ss = dot4(yv[u], yv[u], ss);
  const float rinv = 1.0f / sqrtf(row_sum(ss, red) / (float)D + eps);
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    const int c = (u * blockDim.x + threadIdx.x) * 4;
    if (c >= D) break;
    const float4 v = make_float4(xv[u].x + mult * (yv[u].x * rinv * wv[u].x), xv[u].y + mult * (yv[u].y * rinv * wv[u].y),
                                 xv[u].z + mult * (yv[u].z * rinv * wv[u].z), xv[u].w + mult * (yv[u].w * rinv * wv[u].w));
    put4(x, x16, r * D + c, v);
  }
}

// group == O: one norm over the row (block-wide sum); group < O: one norm per group (a warp per group).
__global__ void __launch_bounds__(256) gated_rmsnorm_kernel(const float* __restrict__ o, const float* __restrict__ gate,
                                                            int ld_gate, const float* __restrict__ w, int wlen, int group,
                                                            float eps, int O, float* __restrict__ out,
                                                            bf16* __restrict__ out16) {
  __shared__ float red[32];
  pdl_launch();
  pdl_wait();
  const size_t r = blockIdx.x;
  const float* orow = o + r * O;
  const float* grow = gate + r * ld_gate;
  if (group >= O) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < O; i += blockDim.x) { const float v = orow[i]; ss = fmaf(v, v, ss); }
    const float rinv = 1.0f / sqrtf(block_sum(ss, red) / (float)O + eps);
    for (int i = threadIdx.x; i < O; i += blockDim.x) {
      const float v = orow[i] * rinv * w[i % wlen] * sigmoid_f(grow[i]);
      out[r * O + i] = v;
      if (out16) out16[r * O + i] = __float2bfloat16_rn(v);
    }
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int g = warp; g * group < O; g += nw) {
    const int base = g * group;
    float ss = 0.f;
    for (int i = lane; i < group; i += 32) { const float v = orow[base + i]; ss = fmaf(v, v, ss); }
    const float rinv = 1.0f / sqrtf(warp_sum(ss) / (float)group + eps);
    for (int i = lane; i < group; i += 32) {
      const float v = orow[base + i] * rinv * w[(base + i) % wlen] * sigmoid_f(grow[base + i]);
      out[r * O + base + i] = v;
      if (out16) out16[r * O + base + i] = __float2bfloat16_rn(v);
    }
  }
}

template <typename KVT>
__global__ void __launch_bounds__(256) qk_norm_cache_kernel(QkNormArgs a) {
  __shared__ float red[32];
  pdl_launch();
  pdl_wait();
  const int r = blockIdx.x;
  const int b = r / a.L, t = r - b * a.L;
  const int pos = *a.pos_ptr + t;
  const float* row = a.proj + (size_t)r * a.ld;
  const int nq = a.HN * a.HD, nk = a.KVHN * a.HD;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nq; i += blockDim.x) { const float v = row[i]; ss = fmaf(v, v, ss); }
  const float rq = 1.0f / sqrtf(block_sum(ss, red) / (float)nq + a.eps);
  if (a.q_out)
    for (int i = threadIdx.x; i < nq; i += blockDim.x) a.q_out[(size_t)r * nq + i] = row[i] * rq * a.wq[i];
  if (a.q16) {  // operand of the tensor-core kernel: the bf16 value of four entries at a time, then what it leaves
    const int n4 = a.HN * a.q16_ld / 4;
    for (int g = threadIdx.x; g < n4; g += blockDim.x) {
      const int h = g * 4 / a.q16_ld, d = g * 4 - h * a.q16_ld;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (d < a.HD) {  // HD is a multiple of 8
        const float* src = row + h * a.HD + d;
        const float* w = a.wq + h * a.HD + d;
        v = make_float4(src[0] * rq * w[0], src[1] * rq * w[1], src[2] * rq * w[2], src[3] * rq * w[3]);
      }
      bf16* dst = a.q16 + ((size_t)r * a.HN + h) * 2 * a.q16_ld + d;
      union { __nv_bfloat162 b[2]; uint2 u; } hi, lo;
      hi.b[0] = __floats2bfloat162_rn(v.x, v.y); hi.b[1] = __floats2bfloat162_rn(v.z, v.w);
      lo.b[0] = __floats2bfloat162_rn(bf16_rest(v.x), bf16_rest(v.y)); lo.b[1] = __floats2bfloat162_rn(bf16_rest(v.z), bf16_rest(v.w));
      *reinterpret_cast<uint2*>(dst) = hi.u;
      *reinterpret_cast<uint2*>(dst + a.q16_ld) = lo.u;
    }
  }
  const float* krow = row + a.k_off;
  ss = 0.f;
  for (int i = threadIdx.x; i < nk; i += blockDim.x) { const float v = krow[i]; ss = fmaf(v, v, ss); }
  const float rk = 1.0f / sqrtf(block_sum(ss, red) / (float)nk + a.eps);
  for (int i = threadIdx.x; i < nk; i += blockDim.x) {
    const int h = i / a.HD, d = i - h * a.HD;
    const size_t ci = (((size_t)b * a.KVHN + h) * a.M + pos) * a.HD + d;
    const float v = krow[i];
    ((KVT*)a.cache_k)[ci] = from_f32<KVT>(v * rk * a.wk[i]);
    ((KVT*)a.cache_v)[ci] = from_f32<KVT>(v);
  }
}

// the same with q and k rows in registers: 2048 rows of 16 + 4 heads of 128: 25.6 -> 13.2 us
template <typename KVT, int NV>
__global__ void __launch_bounds__(256) qk_norm_cache_vec_kernel(QkNormArgs a) {
  __shared__ float red[2][32];
  pdl_launch();
  pdl_wait();
  const int r = blockIdx.x;
  const int b = r / a.L, t = r - b * a.L;
  const int pos = *a.pos_ptr + t;
  const float* row = a.proj + (size_t)r * a.ld;
  const int nq = a.HN * a.HD, nk = a.KVHN * a.HD;
  float4 q[NV], k[NV], wq[NV], wk[NV];
  row_load(row, nq, q);
  row_load(row + a.k_off, nk, k);
  row_load(a.wq, nq, wq);
  row_load(a.wk, nk, wk);
  float sq = 0.f, sk = 0.f;
#pragma unroll
  for (int u = 0; u < NV; ++u) { sq = dot4(q[u], q[u], sq); sk = dot4(k[u], k[u], sk); }
  const float rq = 1.0f / sqrtf(row_sum(sq, red[0]) / (float)nq + a.eps), rk = 1.0f / sqrtf(row_sum(sk, red[1]) / (float)nk + a.eps);
  auto scaled = [](const float4& v, float f, const float4& w) { return make_float4(v.x * f * w.x, v.y * f * w.y, v.z * f * w.z, v.w * f * w.w); };
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    const int c = (u * blockDim.x + threadIdx.x) * 4;
    if (c < nq) {
      const float4 v = scaled(q[u], rq, wq[u]);
      if (a.q_out) *reinterpret_cast<float4*>(a.q_out + (size_t)r * nq + c) = v;
      if (a.q16) {  // operand of the tensor-core kernel: the bf16 values, then what they leave
        const int h = c / a.HD, d = c - h * a.HD;
        bf16* dst = a.q16 + ((size_t)r * a.HN + h) * 2 * a.q16_ld + d;
        put4(nullptr, dst, 0, v);
        put4(nullptr, dst, a.q16_ld, make_float4(bf16_rest(v.x), bf16_rest(v.y), bf16_rest(v.z), bf16_rest(v.w)));
      }
    }
    if (c < nk) {
      const int h = c / a.HD, d = c - h * a.HD;
      const size_t ci = (((size_t)b * a.KVHN + h) * a.M + pos) * a.HD + d;
      const float4 v = scaled(k[u], rk, wk[u]);
      if constexpr (sizeof(KVT) == 2) {
        put4(nullptr, (bf16*)a.cache_k, ci, v);
        put4(nullptr, (bf16*)a.cache_v, ci, k[u]);
      } else {
        put4((float*)a.cache_k, nullptr, ci, v);
        put4((float*)a.cache_v, nullptr, ci, k[u]);
      }
    }
  }
  if (a.q16 && a.q16_ld > a.HD) {  // zeros behind a head's entries, in groups of four
    const int z4 = (a.q16_ld - a.HD) / 4, n = a.HN * 2 * z4;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int hp = i / z4, d = a.HD + (i - hp * z4) * 4;
      put4(nullptr, a.q16 + ((size_t)r * a.HN * 2 + hp) * a.q16_ld, d, make_float4(0.f, 0.f, 0.f, 0.f));
    }
  }
}

template <typename WT>
__global__ void side_mul_kernel(float* __restrict__ g, int n, int rows, const WT* __restrict__ table, int table_ld,
                                int col0, const int32_t* __restrict__ ids, int ids_ld, int ids_off, int L, int vocab,
                                int act, bf16* __restrict__ out16) {
  pdl_launch();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)rows * n) return;
  const int r = (int)(i / n), j = (int)(i - (int64_t)r * n);
  const int b = r / L, t = r - b * L;
  const int id = min(max(ids[(size_t)b * ids_ld + ids_off + t], 0), vocab - 1);
  const float z = g[i];
  const float a = act == GLU_GELU_TANH ? gelu_tanh_ref(z) : silu_ref(z);
  const float v = a * to_f32(table[(size_t)id * table_ld + col0 + j]);
  g[i] = v;
  if (out16) out16[i] = __float2bfloat16_rn(v);
}

// Input of channel c at time t' < 0 of the call comes from the tail [C][taps-1] (oldest first) that earlier calls left.
// The work of a token row is a list of items - a q or k head (convolution + silu + unit length), a v head (convolution +
// silu), a head's decays, the write strengths - and every warp of the row's CTAs (blockIdx.y of them: few rows spread a
// row over several CTAs) takes items round-robin; no item needs another warp.
__global__ void __launch_bounds__(256) delta_prep_kernel(DeltaPrepArgs a) {
  extern __shared__ float sm[];  // [warps][DK] the convolved head a warp works on
  pdl_launch();
  pdl_wait();
  const int r = blockIdx.x;
  const int b = r / a.L, t = r - b * a.L;
  const int nq = a.G * a.DK, nv = a.H * a.DV, C = 2 * nq + nv, T1 = a.taps - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* tail = a.conv_tail + (size_t)b * C * T1;
  float* buf = sm + (size_t)warp * a.DK;
  auto conv = [&](int c) {
    float acc = 0.f;
    for (int j = 0; j < a.taps; ++j) {
      const int tt = t - T1 + j;  // time inside this call; negative: from the tail
      const float xin = tt >= 0 ? a.proj[(size_t)(b * a.L + tt) * a.ld + c] : tail[(size_t)c * T1 + (T1 + tt)];
      acc = fmaf(a.conv_w[(size_t)c * a.taps + j], xin, acc);
      // a call of one token moves the tail on here: this thread alone reads and writes channel c's entries
      if (a.update_tail && j >= 1 && j <= T1) tail[(size_t)c * T1 + (j - 1)] = xin;
    }
    return silu_ref(acc);
  };
  const int n_items = 2 * a.G + 2 * a.H + 1;
  for (int item = blockIdx.y * nw + warp; item < n_items; item += gridDim.y * nw) {
    if (item < 2 * a.G) {  // a q or k head: unit length; q also times DK^-1/2
      float ss = 0.f;
      for (int i = lane; i < a.DK; i += 32) { const float v = conv(item * a.DK + i); buf[i] = v; ss = fmaf(v, v, ss); }
      float rinv = 1.0f / sqrtf(warp_sum(ss) + 1e-6f);
      const bool is_q = item < a.G;
      if (is_q) rinv *= 1.0f / sqrtf((float)a.DK);
      float* dst = is_q ? a.q_out + (size_t)r * nq + (size_t)item * a.DK : a.k_out + (size_t)r * nq + (size_t)(item - a.G) * a.DK;
      for (int i = lane; i < a.DK; i += 32) dst[i] = buf[i] * rinv;  // a lane reads back what it wrote itself
    } else if (item < 2 * a.G + a.H) {
      const int h = item - 2 * a.G;
      for (int i = lane; i < a.DV; i += 32) a.v_out[(size_t)r * nv + (size_t)h * a.DV + i] = conv(2 * nq + h * a.DV + i);
    } else if (item < 2 * a.G + 2 * a.H) {  // decay per key channel of a head
      const int h = item - 2 * a.G - a.H;
      const float rate = expf(a.A_log[h]);
      for (int i = lane; i < a.DK; i += 32) {
        const int c = h * a.DK + i;
        const float lg = -rate * softplus_f(a.dt_in[(size_t)r * a.ld_dt + c] + a.dt_bias[c]);
        a.decay_out[(size_t)r * a.H * a.DK + c] = a.log_decay ? lg : expf(lg);
      }
    } else {
      for (int h = lane; h < a.H; h += 32) a.beta_out[(size_t)r * a.H + h] = sigmoid_f(a.proj[(size_t)r * a.ld + a.beta_off + h]);
    }
  }
}

// Prompts with heads of 128 and 4 taps: a warp takes one item of CONV_TOKENS tokens, a lane four channels, so that a convolution reads
// every input once instead of four times and no value goes through shared memory.  2048 tokens, 16 heads: 103 -> 37 us (134 MB)
__global__ void __launch_bounds__(256) delta_prep_vec_kernel(DeltaPrepArgs a) {
  pdl_launch();
  pdl_wait();
  const int lane = threadIdx.x & 31, c4 = lane * 4, b = blockIdx.z, t0 = blockIdx.x * CONV_TOKENS, n = min(CONV_TOKENS, a.L - t0);
  const int nq = a.G * 128, nv = a.H * a.DV, nvi = nv / 128, C = 2 * nq + nv;
  const int item = blockIdx.y * 8 + (threadIdx.x >> 5);
  const size_t r0 = (size_t)b * a.L + t0;
  if (item < 2 * a.G + nvi) {  // 128 channels: a q head, a k head, a part of a v head
    const int c = item * 128 + c4;
    Conv4 cv;
    cv.load(a.proj + (size_t)b * a.L * a.ld + c, a.ld, a.conv_tail + ((size_t)b * C + c) * 3, a.conv_w + (size_t)c * 4, t0, a.L);
    const bool is_q = item < a.G, unit = item < 2 * a.G;
    float* dst = is_q ? a.q_out + r0 * nq + c : unit ? a.k_out + r0 * nq + (c - nq) : a.v_out + r0 * nv + (c - 2 * nq);
    const int ld = unit ? nq : nv;
    const float mul = is_q ? 1.0f / sqrtf(128.f) : 1.0f;
#pragma unroll
    for (int i = 0; i < CONV_TOKENS; ++i) {
      if (i >= n) break;
      float4 v = cv.at(i, make_float4(0.f, 0.f, 0.f, 0.f));
      v = make_float4(silu_ref(v.x), silu_ref(v.y), silu_ref(v.z), silu_ref(v.w));
      if (unit) {
        const float f = 1.0f / sqrtf(warp_sum(dot4(v, v, 0.f)) + 1e-6f) * mul;
        v = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
      }
      *reinterpret_cast<float4*>(dst + (size_t)i * ld) = v;
    }
  } else if (item < 2 * a.G + nvi + a.H) {  // decay per key channel of a head
    const int h = item - 2 * a.G - nvi, c = h * 128 + c4;
    const float rate = expf(a.A_log[h]);
    const float4 bias = *reinterpret_cast<const float4*>(a.dt_bias + c);
    float4 x[CONV_TOKENS];
#pragma unroll
    for (int i = 0; i < CONV_TOKENS; ++i)
      if (i < n) x[i] = *reinterpret_cast<const float4*>(a.dt_in + (r0 + i) * a.ld_dt + c);
    auto f = [&](float z) { const float lg = -rate * softplus_f(z); return a.log_decay ? lg : expf(lg); };
#pragma unroll
    for (int i = 0; i < CONV_TOKENS; ++i)
      if (i < n)
        *reinterpret_cast<float4*>(a.decay_out + (r0 + i) * a.H * 128 + c) = make_float4(f(x[i].x + bias.x), f(x[i].y + bias.y), f(x[i].z + bias.z), f(x[i].w + bias.w));
  } else if (item == 2 * a.G + nvi + a.H) {
    for (int j = lane; j < n * a.H; j += 32) {
      const size_t r = r0 + j / a.H;
      const int h = j % a.H;
      a.beta_out[r * a.H + h] = sigmoid_f(a.proj[r * a.ld + a.beta_off + h]);
    }
  }
}

// new tail[r] = element L + r of (old tail | the call's L inputs); ascending r never reads what it wrote
__global__ void conv_tail_kernel(float* __restrict__ tail, const float* __restrict__ proj, int ld, int B, int L, int C, int T1) {
  pdl_launch();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B * C) return;
  const int b = i / C, c = i - b * C;
  float* tl = tail + ((size_t)b * C + c) * T1;
  for (int r = 0; r < T1; ++r) {
    const int v = L + r;  // index into the virtual sequence
    tl[r] = v < T1 ? tl[v] : proj[(size_t)(b * L + (v - T1)) * ld + c];
  }
}

// out[r] = x[source row of r] / rms * w, any D; source row = src_rows[r] or r * src_mul + src_add; groups > 1: the row is
// cut into that many equal parts, each over its own root mean square
__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, float eps,
                                                           int D, int src_mul, int src_add, const int32_t* __restrict__ src_rows,
                                                           int groups, float* __restrict__ out, bf16* __restrict__ out16) {
  __shared__ float red[32];
  __shared__ float rg[128];
  pdl_launch();
  pdl_wait();
  const size_t r = blockIdx.x;
  const float* xr = x + (src_rows ? (size_t)src_rows[r] : r * src_mul + src_add) * D;
  const int gs = D / groups;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const int wpg = max(1, nw / groups), gpr = nw / wpg;  // warps per group, groups settled per round
  for (int g0 = 0; g0 < groups; g0 += gpr) {
    const int g = g0 + warp / wpg, sub = warp % wpg;
    float ss = 0.f;
    if (g < groups && warp < gpr * wpg)
      for (int i = sub * 32 + lane; i < gs; i += wpg * 32) { const float v = xr[g * gs + i]; ss = fmaf(v, v, ss); }
    ss = warp_sum(ss);
    __syncthreads();
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    if (g < groups && warp < gpr * wpg && sub == 0 && lane == 0) {
      float tot = 0.f;
      for (int w = 0; w < wpg; ++w) tot += red[warp + w];
      rg[g] = 1.0f / sqrtf(tot / (float)gs + eps);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    const float v = xr[i] * rg[i / gs] * w[i];
    out[r * D + i] = v;
    if (out16) out16[r * D + i] = __float2bfloat16_rn(v);
  }
}

// eight values per thread: 2048 x 2048 19.4 -> 5.3 us
__global__ void to_bf16_vec_kernel(const float* __restrict__ in, int64_t n8, bf16* __restrict__ out) {
  pdl_launch();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  const float4 a = reinterpret_cast<const float4*>(in)[2 * i], b = reinterpret_cast<const float4*>(in)[2 * i + 1];
  union { __nv_bfloat162 h[4]; uint4 q; } o;
  o.h[0] = __floats2bfloat162_rn(a.x, a.y); o.h[1] = __floats2bfloat162_rn(a.z, a.w);
  o.h[2] = __floats2bfloat162_rn(b.x, b.y); o.h[3] = __floats2bfloat162_rn(b.z, b.w);
  reinterpret_cast<uint4*>(out)[i] = o.q;
}

__global__ void to_bf16_kernel(const float* __restrict__ in, int64_t n, bf16* __restrict__ out) {
  pdl_launch();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16_rn(in[i]);
}

__global__ void add_one_kernel(float* __restrict__ p, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] += 1.0f;
}

}  // namespace

static int row_threads(int n) { return n >= 1024 ? 256 : n >= 256 ? 128 : 64; }

cudaError_t launch_resid_postnorm(float* x, const float* y, const float* w, float mult, float eps, int rows, int D,
                                  bf16* x16, cudaStream_t s) {
  const RowShape sh = row_shape(D);
  if (sh.nv && sh.nv <= 4 && aligned16(x) && aligned16(y) && aligned16(w) && aligned8(x16))
    return ROW_SWITCH(sh.nv, launch_k(resid_postnorm_vec_kernel<NV>, dim3(rows), dim3(sh.threads), 0, s, x, y, w, mult, eps, D, x16));
  return launch_k(resid_postnorm_kernel, dim3(rows), dim3(row_threads(D)), 0, s, x, y, w, mult, eps, D, x16);
}

cudaError_t launch_gated_rmsnorm(const float* o, const float* gate, int ld_gate, const float* w, int wlen, int group,
                                 float eps, int rows, int O, float* out, bf16* out16, cudaStream_t s) {
  const MixOutArgs mo{o, O, nullptr, nullptr, 1, gate, ld_gate, 0, 0, w, wlen, group, eps, 1.0f, out, out16, O, nullptr, nullptr};
  if (mix_out_vec_supported(mo)) return launch_mix_out_vec(mo, rows, s);  // any number of rows: portions of a prompt add up alike
  const int threads = group >= O ? row_threads(O) : std::min(256, std::max(32, 32 * (O / group)));
  return launch_k(gated_rmsnorm_kernel, dim3(rows), dim3(threads), 0, s, o, gate, ld_gate, w, wlen, group, eps, O, out, out16);
}

cudaError_t launch_qk_norm_cache(const QkNormArgs& a, int rows, bool kv_bf16, cudaStream_t s) {
  const RowShape sh = row_shape(a.HN * a.HD);
  if (sh.nv && sh.nv <= 4 && a.KVHN <= a.HN && a.HD % 4 == 0 && a.ld % 4 == 0 && a.k_off % 4 == 0 && (!a.q16 || a.q16_ld % 4 == 0) && aligned16(a.proj) &&
      aligned16(a.wq) && aligned16(a.wk) && aligned16(a.q_out) && aligned8(a.q16) && aligned16(a.cache_k) && aligned16(a.cache_v))
    return ROW_SWITCH(sh.nv, kv_bf16 ? launch_k(qk_norm_cache_vec_kernel<bf16, NV>, dim3(rows), dim3(sh.threads), 0, s, a)
                                     : launch_k(qk_norm_cache_vec_kernel<float, NV>, dim3(rows), dim3(sh.threads), 0, s, a));
  const int threads = row_threads(a.HN * a.HD);
  if (kv_bf16) return launch_k(qk_norm_cache_kernel<bf16>, dim3(rows), dim3(threads), 0, s, a);
  return launch_k(qk_norm_cache_kernel<float>, dim3(rows), dim3(threads), 0, s, a);
}

cudaError_t launch_side_mul(float* g, int n, int rows, const void* table, bool table_bf16, int table_ld, int col0,
                            const int32_t* ids, int ids_ld, int ids_off, int L, int vocab, int act, bf16* out16,
                            cudaStream_t s) {
  const int64_t tot = (int64_t)rows * n;
  const dim3 grid((unsigned)((tot + 255) / 256));
  if (table_bf16)
    return launch_k(side_mul_kernel<bf16>, grid, dim3(256), 0, s, g, n, rows, (const bf16*)table, table_ld, col0, ids, ids_ld, ids_off, L, vocab, act, out16);
  return launch_k(side_mul_kernel<float>, grid, dim3(256), 0, s, g, n, rows, (const float*)table, table_ld, col0, ids, ids_ld, ids_off, L, vocab, act, out16);
}

cudaError_t launch_delta_prep(const DeltaPrepArgs& a, int rows, cudaStream_t s) {
  if (a.update_tail && a.L != 1) return cudaErrorInvalidValue;
  if (rows > 8 && a.L > 1 && a.taps == 4 && a.DK == 128 && (a.H * a.DV) % 128 == 0 && a.ld % 4 == 0 && a.ld_dt % 4 == 0 && rows % a.L == 0 && rows / a.L <= 65535 &&
      aligned16(a.proj) && aligned16(a.dt_in) && aligned16(a.conv_w) && aligned16(a.dt_bias) && aligned16(a.q_out) && aligned16(a.k_out) && aligned16(a.v_out) &&
      aligned16(a.decay_out)) {
    const int items = 2 * a.G + a.H * a.DV / 128 + a.H + 1;
    return launch_k(delta_prep_vec_kernel, dim3((a.L + CONV_TOKENS - 1) / CONV_TOKENS, (items + 7) / 8, rows / a.L), dim3(256), 0, s, a);
  }
  const size_t smem = (size_t)8 * a.DK * sizeof(float);
  if (const cudaError_t e = allow_smem(delta_prep_kernel, smem)) return e;
  const int items = 2 * a.G + 2 * a.H + 1;
  const int parts = rows <= 8 ? std::max(1, std::min(32, (items + 7) / 8)) : 1;  // few rows: a row's items spread over CTAs
  return launch_k(delta_prep_kernel, dim3(rows, parts), dim3(256), smem, s, a);
}

cudaError_t launch_conv_tail(float* tail, const float* proj, int ld, int B, int L, int C, int T1, cudaStream_t s) {
  if (T1 <= 0) return cudaSuccess;
  return launch_k(conv_tail_kernel, dim3((B * C + 127) / 128), dim3(128), 0, s, tail, proj, ld, B, L, C, T1);
}

cudaError_t launch_rmsnorm_rows(const float* x, const float* w, float eps, int rows, int D, int src_mul, int src_add,
                                const int32_t* src_rows, float* out, bf16* out16, cudaStream_t s, int groups) {
  if (groups < 1 || groups > 128 || D % groups != 0) return cudaErrorInvalidValue;
  const NormRowsArgs na{x, w, eps, 0, D, groups, src_mul, src_add, src_rows, nullptr, nullptr, 1, out, out16};
  if (norm_rows_supported(na)) return launch_norm_rows(na, rows, s);
  return launch_k(rmsnorm_rows_kernel, dim3(rows), dim3(row_threads(D)), 0, s, x, w, eps, D, src_mul, src_add, src_rows, groups, out, out16);
}

cudaError_t launch_to_bf16(const float* in, int64_t n, bf16* out, cudaStream_t s) {
  if (n % 8 == 0 && aligned16(in) && aligned16(out))
    return launch_k(to_bf16_vec_kernel, dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0, s, in, n / 8, out);
  return launch_k(to_bf16_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, s, in, n, out);
}

cudaError_t launch_add_one(float* p, int n, cudaStream_t s) {
  add_one_kernel<<<(n + 255) / 256, 256, 0, s>>>(p, n);
  return cudaGetLastError();
}
