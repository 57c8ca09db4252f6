// Rows of fp32 values held in registers: a CTA per row, thread i takes the four values at (u * blockDim + i) * 4, u < NV.
// Every operand is read once, 16 bytes at a time, and all loads of a row are in flight before its sums - the row kernels built on
// this are bound by their bytes (or, with a few rows, by one load and one reduction), not by a chain of short loads.
#pragma once
#include <stdint.h>

#include "common.cuh"

struct RowShape { int threads, nv; };  // nv 0: not a row for these kernels
inline RowShape row_shape(int D) {
  if (D < 4 || D % 4) return {0, 0};
  for (int nv = 1; nv <= 8; nv *= 2) {
    const int t = ((D / 4 + nv - 1) / nv + 31) / 32 * 32;
    if (t <= 256) return {t, nv};
  }
  return {0, 0};
}
inline bool aligned16(const void* p) { return !((uintptr_t)p & 15); }
inline bool aligned8(const void* p) { return !((uintptr_t)p & 7); }
// the expression with NV as the shape's constant
#define ROW_SWITCH(nv, ...)                                    \
  [&] {                                                        \
    switch (nv) {                                              \
      case 1: { constexpr int NV = 1; return __VA_ARGS__; }    \
      case 2: { constexpr int NV = 2; return __VA_ARGS__; }    \
      case 4: { constexpr int NV = 4; return __VA_ARGS__; }    \
      default: { constexpr int NV = 8; return __VA_ARGS__; }   \
    }                                                          \
  }()

template <int NV>
__device__ __forceinline__ void row_load(const float* p, int D, float4 (&v)[NV]) {
#pragma unroll
  for (int u = 0; u < NV; ++u) {
    const int c = (u * blockDim.x + threadIdx.x) * 4;
    v[u] = c < D ? *reinterpret_cast<const float4*>(p + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float s) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}
// four values, and their bf16 mirror (either pointer may be null)
__device__ __forceinline__ void put4(float* out, bf16* out16, size_t i, const float4& v) {
  if (out) *reinterpret_cast<float4*>(out + i) = v;
  if (out16) {
    union { __nv_bfloat162 h[2]; uint2 q; } o;
    o.h[0] = __floats2bfloat162_rn(v.x, v.y);
    o.h[1] = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(out16 + i) = o.q;
  }
}
// sum over the CTA, the same in every thread; red: 32 floats of shared memory
__device__ __forceinline__ float row_sum(float v, float* red) {
  v = warp_sum(v);
  __syncthreads();  // red may still be read from a call before
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
  return t;
}

// Causal convolution over time of four adjacent channels, CONV_TOKENS tokens at a time: every input is read once per call of this
// (three rows of overlap), weights once.  x: the four channels' column in the projection's row of the sequence's first token; tail:
// their 3 older inputs [channel][3], oldest first; w: [channel][4], last tap = current token.
constexpr int CONV_TOKENS = 8;
struct Conv4 {
  float4 in[CONV_TOKENS + 3];
  float4 w[4];  // per channel
  __device__ __forceinline__ void load(const float* x, int ld, const float* tail, const float* wp, int t0, int L) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(wp + 4 * i);
#pragma unroll
    for (int i = 0; i < CONV_TOKENS + 3; ++i) {
      const int t = t0 - 3 + i;
      if (t >= L) in[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      else if (t >= 0) in[i] = *reinterpret_cast<const float4*>(x + (size_t)t * ld);
      else in[i] = make_float4(tail[3 + t], tail[3 + 3 + t], tail[6 + 3 + t], tail[9 + 3 + t]);
    }
  }
  // token t0 + i, starting from bias
  __device__ __forceinline__ float4 at(int i, const float4& bias) const {
    auto one = [](const float4& k, float b, float x0, float x1, float x2, float x3) { return fmaf(k.w, x3, fmaf(k.z, x2, fmaf(k.y, x1, fmaf(k.x, x0, b)))); };
    return make_float4(one(w[0], bias.x, in[i].x, in[i + 1].x, in[i + 2].x, in[i + 3].x), one(w[1], bias.y, in[i].y, in[i + 1].y, in[i + 2].y, in[i + 3].y),
                       one(w[2], bias.z, in[i].z, in[i + 1].z, in[i + 2].z, in[i + 3].z), one(w[3], bias.w, in[i].w, in[i + 1].w, in[i + 2].w, in[i + 3].w));
  }
};
