// fp32 projections of many rows on the 5th-generation tensor cores without giving up fp32's precision: C = A W^T with fp32 A and
// W [N, K] fp32 or bf16.  Every fp32 value is cut into three bf16 parts of 8 significant bits each, x = x1 + x2 + x3, by truncation,
// inside the kernel (exact from 2^-110 up: the third part of a smaller number ends at bf16's smallest, 2^-133): TMA brings raw fp32
// tiles, converter warps write the parts as operand tiles, and one thread
// issues the products of the parts whose order is above 2^-24,
//   a1 b1 | a1 b2 + a2 b1 + a2 b2 + a1 b3 + a3 b1          (W in bf16: a1 w | a2 w + a3 w),
// the leading one and the corrections into two TMEM accumulators.  The tensor core drops the bits below an accumulator's last one
// at every instruction (a drift of ~0.5 ulp each, 3.5e-6 relative over K = 4096 with the 3xTF32 scheme of gemm_tc.cu), so an
// accumulator takes only 128 summed terms (8 instructions); the converter warps then add it to running fp32 sums in registers.
// 600 x 4096 x 1024: 87 us (58 TFLOP/s of fp32 products), the FFMA tiles it replaces 350 us; measured per rule in layerlist.cu (ll_linear).
//
// One 128 x 128 tile per CTA and turn, persistent; 320 threads:
//   warp 0: TMA   warp 1: TMEM + MMA issue   warps 2 - 9: conversion, running sums, epilogue
// A step is 32 values of K.  The parts' tiles hold 64 (128-byte swizzled rows); their halves are two buffers of a ring, so that a
// step is converted while the previous one is multiplied.  The products are not the bound: 12 of 64 cycles per
// step (mma_probe.cu; the tensor pipe counts 22 - 28 % of the cycles at 600 rows, tiles' ends included), against ~600 issue slots of
// conversion per scheduler and shared memory, whose bandwidth raw tiles, parts and the products' reads share; a 256-wide tile would
// read less but its parts and raw tiles do not fit together.
// An infinite operand leaves NaN behind (its parts are inf, NaN, NaN; inf times a zero part is NaN too): sums that end as NaN are
// taken again as a plain chain of fp32 products, so that an infinity gives what it gives there.
// Where both operands were cut beforehand (OP_PLANES: matrices once at load time, inputs by cut_rows_kernel; ll_cut_operands has the rule)
// TMA brings the parts themselves, three planes a copy, and nothing is converted: 24 products per 64 values of K, bound by shared memory,
// whose bandwidth the arriving 96 KB and the products' reads share (~2600 cycles, of which the products take 1536).  600 x 4096 x 1024:
// 64.7 -> 43.4 us, 600 x 1024 x 4096 52.3 -> 37.6, 600 x 1024 x 1024 23 -> 18.8; the same bits.
// Every wait is bounded: one that runs out sets a flag, all warps run on without waiting, and the host reports an error.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "gemm_tc.h"

namespace {

constexpr int TILE = 128, STEP = 32, CHUNK = 4;          // tile edge; values of K per step; steps per accumulator turn
constexpr int HALF = TILE * 128;                         // bytes of a 128-row tile of 128-byte rows
constexpr int THREADS = 320, RAW = 4, WST = 3;        // raw tiles, and weight tiles of the bf16 form, in flight

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, volatile int* fail) {
  for (uint32_t spins = 0; spins < (1u << 20); ++spins) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return;
    if ((spins & 63) == 63 && *fail) return;
  }
  *fail = 1;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(tm), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TILE >> 3) << 17) | ((128u >> 4) << 24);  // bf16 x bf16 -> fp32, 128 x 128
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accum) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(d), "l"(a), "l"(b), "r"(IDESC), "r"(accum) : "memory");
}
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
// K-major, 128-byte-swizzled operand tile: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// eight fp32 values -> three 16-byte pieces of bf16 parts; every subtraction is exact
__device__ __forceinline__ void cut8(const float4& x, const float4& y, uint4& p1, uint4& p2, uint4& p3) {
  const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  uint32_t* o1 = reinterpret_cast<uint32_t*>(&p1);
  uint32_t* o2 = reinterpret_cast<uint32_t*>(&p2);
  uint32_t* o3 = reinterpret_cast<uint32_t*>(&p3);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = v[2 * i], b = v[2 * i + 1];
    const float ra = a - __uint_as_float(__float_as_uint(a) & 0xffff0000u), rb = b - __uint_as_float(__float_as_uint(b) & 0xffff0000u);
    const float sa = ra - __uint_as_float(__float_as_uint(ra) & 0xffff0000u), sb = rb - __uint_as_float(__float_as_uint(rb) & 0xffff0000u);
    o1[i] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
    o2[i] = __byte_perm(__float_as_uint(ra), __float_as_uint(rb), 0x7632);
    o3[i] = __byte_perm(__float_as_uint(sa), __float_as_uint(sb), 0x7632);
  }
}

// a . w in fp32, until it is NaN
template <typename WT>
__device__ float plain_dot(const float* a, const WT* w, int K) {
  float s = 0.f;
  for (int k = 0; k < K && s == s; ++k) s = fmaf(a[k], to_f32(w[k]), s);
  return s;
}

// how the operands come: both fp32, W in bf16, or both cut beforehand (three planes each, GemmF32Args::planes)
enum Operands : int { OP_F32 = 0, OP_W16 = 1, OP_PLANES = 2 };
template <int OP> constexpr int raw_bytes() { return OP == OP_W16 ? HALF : 2 * HALF; }
constexpr int BLOCK = 6 * HALF, PST = 2;  // planes: a block of 64 values of K, three parts of both operands; blocks in flight
template <int OP> constexpr int smem_bytes() {
  return OP == OP_PLANES ? 1024 + PST * BLOCK + 512 : 1024 + 3 * HALF + (OP == OP_W16 ? WST : 3) * HALF + RAW * raw_bytes<OP>() + 512;
}

template <int OP, int EPI>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, int rows, int N, int K, int ksplit, float* part,
                int* tile_cnt, int* err, const float* A, int lda, const void* W, EpiArgs e) {
  constexpr bool WB16 = OP == OP_W16, PLANES = OP == OP_PLANES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t sA = (raw + 1023u) & ~1023u, sW = sA + 3 * HALF, sR = sW + (WB16 ? WST : 3) * HALF, bars = PLANES ? sA + PST * BLOCK : sR + RAW * raw_bytes<OP>();
  uint8_t* base = smem_raw + (sA - raw);
  const uint32_t r_full = bars, r_empty = r_full + 8 * RAW, h_full = r_empty + 8 * RAW, h_empty = h_full + 16, w_full = h_empty + 16,
                 w_empty = w_full + 8 * WST, a_full = w_empty + 8 * WST, a_empty = a_full + 16, slot = a_empty + 16;
  uint32_t* slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (slot - raw));
  volatile int* fail = reinterpret_cast<volatile int*>(slot_ptr + 1);
  int* last_flag = reinterpret_cast<int*>(slot_ptr + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch();
  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA));
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmW));
    *fail = 0;
    for (int s = 0; s < RAW; ++s) { mbar_init(r_full + 8 * s, 1); mbar_init(r_empty + 8 * s, PLANES ? 1 : 8); }
    for (int s = 0; s < WST; ++s) { mbar_init(w_full + 8 * s, 1); mbar_init(w_empty + 8 * s, 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(h_full + 8 * s, 8); mbar_init(h_empty + 8 * s, 1);
      mbar_init(a_full + 8 * s, 1); mbar_init(a_empty + 8 * s, 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(slot));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot_ptr;
  pdl_wait();
  const int tiles_m = (rows + TILE - 1) / TILE, tiles_n = (N + TILE - 1) / TILE, ntiles_mn = tiles_m * tiles_n, ntiles = ntiles_mn * ksplit;
  const int blocks = (K + 63) / 64, per = (blocks + ksplit - 1) / ksplit;  // K in blocks of 64 = two steps (the surplus reads zeros)
  // steps [0, n) of tile t: K values k0 + 32 s
  auto slice = [&](int t, int& k0, int& n) {
    const int ks = t / ntiles_mn, b0 = ks * per, b1 = min(blocks, b0 + per);
    k0 = b0 * 64;
    n = 2 * (b1 - b0);
  };

  if (PLANES && warp == 0) {  // ---------------- TMA; the issuing warps run their loops whole, one elected lane issues
    uint32_t st = 0, ph = 1;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      const int tmn = t % ntiles_mn, m0 = (tmn % tiles_m) * TILE, n0 = (tmn / tiles_m) * TILE;
      int k0, n;
      slice(t, k0, n);
      for (int b = 0; b < n / 2; ++b) {
        mbar_wait(r_empty + 8 * st, ph, fail);
        if (elect_one()) {
          const uint32_t dst = sA + st * BLOCK, bar = r_full + 8 * st;
          mbar_expect_tx(bar, BLOCK);
          tma_load_3d(dst, &tmA, k0 + b * 64, m0, 0, bar);
          tma_load_3d(dst + 3 * HALF, &tmW, k0 + b * 64, n0, 0, bar);
        }
        __syncwarp();
        if (++st == PST) { st = 0; ph ^= 1; }
      }
    }
  } else if (PLANES && warp == 1) {  // ---------------- products
    constexpr uint64_t PART = HALF >> 4;
    uint32_t st = 0, ph = 0, ci = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      int k0, n;
      slice(t, k0, n);
      n /= 2;
      for (int b = 0; b < n; ++b) {
        const uint32_t buf = ci & 1, turn = b & 1;  // an accumulator takes two blocks, 128 terms of each kind
        if (!turn && ci >= 2) mbar_wait(a_empty + 8 * buf, (ci / 2 - 1) & 1, fail);
        mbar_wait(r_full + 8 * st, ph, fail);
        tc_fence_after();
        if (elect_one()) {
          const uint32_t lead = tmem + buf * 256, corr = lead + TILE;
          const uint64_t da = desc_sw128(sA + st * BLOCK), dw = da + 3 * PART;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint64_t a = da + kk * 2, w = dw + kk * 2;
            const uint32_t go = turn | kk ? 1u : 0u;
            mma(lead, a, w, go);
            mma(corr, a, w + PART, go);
            mma(corr, a + PART, w, 1u);
            mma(corr, a + PART, w + PART, 1u);
            mma(corr, a, w + 2 * PART, 1u);
            mma(corr, a + 2 * PART, w, 1u);
          }
          tc_commit(r_empty + 8 * st);
          if (turn || b == n - 1) tc_commit(a_full + 8 * buf);
        }
        __syncwarp();
        if (turn || b == n - 1) ++ci;
        if (++st == PST) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 0) {
    if (lane == 0) {  // ---------------- TMA
      uint32_t it = 0, wt = 0;
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int tmn = t % ntiles_mn, m0 = (tmn % tiles_m) * TILE, n0 = (tmn / tiles_m) * TILE;
        int k0, n;
        slice(t, k0, n);
        for (int s = 0; s < n; ++s, ++it) {
          if (WB16 && !(s & 1)) {
            const uint32_t st = wt % WST;
            if (wt >= WST) mbar_wait(w_empty + 8 * st, (wt / WST - 1) & 1, fail);
            mbar_expect_tx(w_full + 8 * st, HALF);
            tma_load_2d(sW + st * HALF, &tmW, k0 + s * STEP, n0, w_full + 8 * st);
            ++wt;
          }
          const uint32_t st = it % RAW;
          if (it >= RAW) mbar_wait(r_empty + 8 * st, (it / RAW - 1) & 1, fail);
          mbar_expect_tx(r_full + 8 * st, raw_bytes<OP>());
          tma_load_2d(sR + st * raw_bytes<OP>(), &tmA, k0 + s * STEP, m0, r_full + 8 * st);
          if (!WB16) tma_load_2d(sR + st * raw_bytes<OP>() + HALF, &tmW, k0 + s * STEP, n0, r_full + 8 * st);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ---------------- products
      const uint64_t da = desc_sw128(sA), dw = desc_sw128(sW);
      constexpr uint64_t PART = HALF >> 4;
      uint32_t it = 0, wt = 0, ci = 0;
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        int k0, n;
        slice(t, k0, n);
        for (int s = 0; s < n; ++s, ++it) {
          const uint32_t h = it & 1, buf = ci & 1;
          if (s % CHUNK == 0 && ci >= 2) mbar_wait(a_empty + 8 * buf, (ci / 2 - 1) & 1, fail);
          if (WB16 && h == 0) mbar_wait(w_full + 8 * (wt % WST), (wt / WST) & 1, fail);
          mbar_wait(h_full + 8 * h, (it >> 1) & 1, fail);
          tc_fence_after();
          const uint32_t lead = tmem + buf * 256, corr = lead + TILE;
          const uint64_t wd = WB16 ? dw + (wt % WST) * PART : dw;
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const uint64_t a = da + (h * 2 + kk) * 2, w = wd + (h * 2 + kk) * 2;
            const uint32_t go = (s % CHUNK) | kk ? 1u : 0u;
            mma(lead, a, w, go);
            if (WB16) {
              mma(corr, a + PART, w, go);
              mma(corr, a + 2 * PART, w, 1u);
            } else {
              mma(corr, a, w + PART, go);
              mma(corr, a + PART, w, 1u);
              mma(corr, a + PART, w + PART, 1u);
              mma(corr, a, w + 2 * PART, 1u);
              mma(corr, a + 2 * PART, w, 1u);
            }
          }
          tc_commit(h_empty + 8 * h);
          if (WB16 && h == 1) { tc_commit(w_empty + 8 * (wt % WST)); ++wt; }
          if (s % CHUNK == CHUNK - 1 || s == n - 1) { tc_commit(a_full + 8 * buf); ++ci; }
        }
      }
    }
  } else {  // ---------------- conversion, running sums, epilogue
    const int ct = threadIdx.x - 64, quarter = warp & 3, c0 = ((warp - 2) >> 2) * 64;  // TMEM lanes and columns of this warp
    const uint32_t tl = tmem + ((uint32_t)(quarter * 32) << 16) + c0;
    uint32_t it = 0, pi = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      const int tmn = t % ntiles_mn, m0 = (tmn % tiles_m) * TILE, n0 = (tmn / tiles_m) * TILE;
      int k0, n;
      slice(t, k0, n);
      float run[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) run[j] = 0.f;
      auto promote = [&]() {
        const uint32_t buf = pi & 1;
        mbar_wait(a_full + 8 * buf, (pi >> 1) & 1, fail);
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          float x[32], y[32];
          tmem_ld32_issue(tl + buf * 256 + c, x);
          tmem_ld32_issue(tl + buf * 256 + TILE + c, y);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; ++j) run[c + j] += x[j] + y[j];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(a_empty + 8 * buf);
        ++pi;
      };
#pragma unroll 1
      for (int s = 0; s < (PLANES ? 0 : n); ++s, ++it) {
        const uint32_t st = it % RAW, h = it & 1;
        mbar_wait(r_full + 8 * st, (it / RAW) & 1, fail);
        if (it >= 2) mbar_wait(h_empty + 8 * h, ((it >> 1) - 1) & 1, fail);
        // a thread: a row of 32 values (W bf16: half a row of A); 16-byte pieces swizzled inside the 128-byte rows on both sides
        const int r = WB16 ? ct >> 1 : ct & 127, op = WB16 ? 0 : ct >> 7, q0 = WB16 ? (ct & 1) * 4 : 0;
        const uint8_t* src = base + (sR - sA) + st * raw_bytes<OP>() + op * HALF + r * 128;
        uint8_t* dst = base + op * 3 * HALF + r * 128;
#pragma unroll
        for (int q = 0; q < (WB16 ? 4 : 8); q += 2) {
          const int qq = q0 + q;
          const float4 x = *reinterpret_cast<const float4*>(src + ((qq ^ (r & 7)) << 4)), y = *reinterpret_cast<const float4*>(src + (((qq + 1) ^ (r & 7)) << 4));
          uint4 p1, p2, p3;
          cut8(x, y, p1, p2, p3);
          const int o = ((h * 4 + (qq >> 1)) ^ (r & 7)) << 4;
          *reinterpret_cast<uint4*>(dst + o) = p1;
          *reinterpret_cast<uint4*>(dst + HALF + o) = p2;
          *reinterpret_cast<uint4*>(dst + 2 * HALF + o) = p3;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) { mbar_arrive(r_empty + 8 * st); mbar_arrive(h_full + 8 * h); }
        if (s % CHUNK == CHUNK - 1 && s >= CHUNK) promote();  // the turn before this one: its products are long issued
      }
      for (int left = (n + CHUNK - 1) / CHUNK - (PLANES ? 0 : max(0, n / CHUNK - 1)); left > 0; --left) promote();
      const int m = m0 + quarter * 32 + lane, nc = n0 + c0;
      if (ksplit > 1) {
        // publish this slice's sums; the slice that arrives last adds all of them in slice order (the result does not depend on timing)
        // scratch [k slice][output tile][column / 4][row of the tile] float4: a warp's rows are contiguous
        const size_t slice_len = (size_t)ntiles_mn * (TILE / 4) * TILE;
        float4* p = reinterpret_cast<float4*>(part) + ((size_t)tmn * (TILE / 4) + c0 / 4) * TILE + quarter * 32 + lane;
        const int ks = t / ntiles_mn;
        if (m < rows)
#pragma unroll
          for (int j = 0; j < 64; j += 4) __stcg(p + ks * slice_len + (size_t)(j / 4) * TILE, make_float4(run[j], run[j + 1], run[j + 2], run[j + 3]));
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (ct == 0) {
          int old;
          asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(tile_cnt + tmn) : "memory");
          *last_flag = old == ksplit - 1;
          if (old == ksplit - 1) tile_cnt[tmn] = 0;  // ready for the next launch
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const bool is_last = *last_flag != 0;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (!is_last) continue;
        if (m < rows) {
#pragma unroll
          for (int j = 0; j < 64; ++j) run[j] = 0.f;
          for (int k2 = 0; k2 < ksplit; ++k2) {
            float4 q[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) q[j] = __ldcg(p + k2 * slice_len + (size_t)j * TILE);
#pragma unroll
            for (int j = 0; j < 16; ++j) { run[4 * j] += q[j].x; run[4 * j + 1] += q[j].y; run[4 * j + 2] += q[j].z; run[4 * j + 3] += q[j].w; }
          }
        }
      }
      if (m >= rows) continue;
      uint64_t odd = 0;
#pragma unroll
      for (int j = 0; j < 64; ++j) odd |= (uint64_t)(run[j] != run[j]) << j;
      for (; odd; odd &= odd - 1) {
        const int c = __ffsll(odd) - 1;
        if (nc + c >= N) break;
        const float v = plain_dot(A + (size_t)m * lda, reinterpret_cast<const std::conditional_t<WB16, bf16, float>*>(W) + (size_t)(nc + c) * K, K);
#pragma unroll
        for (int j = 0; j < 64; ++j) run[j] = j == c ? v : run[j];
      }
      const bool plain = !e.out_lo && !e.out_bf16 && !e.glu_w && !(e.ld_out & 3) && !(N & 3);
#pragma unroll
      for (int j = 0; j < 64; j += 4) {
        const int col = nc + j;
        if (col >= N) break;
        if (plain && EPI != EPI_SWIGLU) {
          float4 v = make_float4(run[j], run[j + 1], run[j + 2], run[j + 3]);
          const size_t o = (size_t)m * e.ld_out + col;
          if (EPI == EPI_RESID) {
            const float4 x = *reinterpret_cast<const float4*>(e.resid + o);
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
          } else if (e.unary) {
            v.x = unary_act(e.unary, v.x); v.y = unary_act(e.unary, v.y); v.z = unary_act(e.unary, v.z); v.w = unary_act(e.unary, v.w);
          }
          *reinterpret_cast<float4*>(e.out + o) = v;
        } else if (plain) {
          const float2 v = make_float2(glu_pair<false>(e, run[j], run[j + 1]), glu_pair<false>(e, run[j + 2], run[j + 3]));
          *reinterpret_cast<float2*>(e.out + (size_t)m * e.ld_out + (col >> 1)) = v;
        } else {
          epilogue_pair<float>(EPI, e, m, col, run[j], run[j + 1], col + 1 < N);
          if (col + 2 < N) epilogue_pair<float>(EPI, e, m, col + 2, run[j + 2], run[j + 3], col + 3 < N);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *fail) {
    if (err) *err = 1;
    __nanosleep(1000000);  // copies still in flight land before the shared memory is given up
  }
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

template <int OP, int EPI>
cudaError_t launch_t(const GemmF32Args& a, cudaStream_t s) {
  auto kern = gemm_f32_kernel<OP, EPI>;
  static bool done[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!done[dev & 15]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<OP>());
    if (e != cudaSuccess) return e;
    done[dev & 15] = true;
  }
  const bool pl = OP == OP_PLANES;
  const CUtensorMap* ma = pl ? tc_get_planes_map(a.A_planes, a.rows, a.K, TILE, a.a_plane) : tc_get_map(a.A, false, a.rows, a.K, TILE, a.lda);
  const CUtensorMap* mw = pl ? tc_get_planes_map(a.W_planes, a.N, a.K, TILE, a.w_plane) : tc_get_map(a.W, OP == OP_W16, a.N, a.K, TILE);
  if (!ma || !mw) return cudaErrorInvalidValue;
  static int n_sm[16] = {0};
  if (!n_sm[dev & 15]) cudaDeviceGetAttribute(&n_sm[dev & 15], cudaDevAttrMultiProcessorCount, dev);
  const int sms = n_sm[dev & 15] > 0 ? n_sm[dev & 15] : 148;
  const int tm = (a.rows + TILE - 1) / TILE, tn = (a.N + TILE - 1) / TILE, tiles = tm * tn, blocks = (a.K + 63) / 64;
  // K split over CTAs: the rounds of the machine times a slice's length, with ~2 blocks of 64 for a slice's start, publication and end
  int ksplit = 1;
  if (a.part && a.tile_cnt && tiles <= a.tile_cnt_len) {
    long best = 0;
    for (int ks = 1; ks <= 8; ++ks) {
      const int per = (blocks + ks - 1) / ks;
      if (ks > 1 && (per < 2 || (ks - 1) * per >= blocks || (size_t)tm * tn * TILE * TILE * 4 * ks > a.part_bytes)) continue;
      const long cost = (long)((tiles * ks + sms - 1) / sms) * (per + 2);
      if (!best || cost < best) { best = cost; ksplit = ks; }
    }
  }
  return launch_k(kern, dim3(std::min(tiles * ksplit, sms)), dim3(THREADS), (size_t)smem_bytes<OP>(), s, *ma, *mw, a.rows, a.N, a.K, ksplit, a.part,
                  a.tile_cnt, a.err, a.A, a.lda ? a.lda : a.K, a.W, a.e);
}

template <int OP>
cudaError_t launch_e(const GemmF32Args& a, cudaStream_t s) {
  switch (a.epi) {
    case EPI_STORE: return launch_t<OP, EPI_STORE>(a, s);
    case EPI_RESID: return launch_t<OP, EPI_RESID>(a, s);
    case EPI_SWIGLU: return launch_t<OP, EPI_SWIGLU>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

bool gemm_f32_supported(const GemmF32Args& a) {
  if (a.epi != EPI_STORE && a.epi != EPI_RESID && a.epi != EPI_SWIGLU) return false;
  const int lda = a.lda ? a.lda : a.K;
  if ((((uintptr_t)a.A | (uintptr_t)a.W) & 15) || lda % 4 || a.K % (a.w_bf16 ? 8 : 4)) return false;  // 16-byte rows of the tensor maps
  // 16-byte rows of what the epilogue reads and writes
  return !(((uintptr_t)a.e.out | (uintptr_t)a.e.resid) & 15) && tc_gemm_supported(8);
}

cudaError_t launch_gemm_f32(const GemmF32Args& a, cudaStream_t s) {
  if (!gemm_f32_supported(a)) return cudaErrorInvalidValue;
  if (!a.w_bf16 && a.A_planes && a.W_planes) {
    if (a.K % 8 || a.a_plane % 8 || a.w_plane % 8 || (((uintptr_t)a.A_planes | (uintptr_t)a.W_planes) & 15)) return cudaErrorInvalidValue;
    return launch_e<OP_PLANES>(a, s);
  }
  return a.w_bf16 ? launch_e<OP_W16>(a, s) : launch_e<OP_F32>(a, s);
}

bool gemm_f32_planes_supported(const void* W_planes, int64_t w_plane, int K) { return W_planes && K % 8 == 0 && w_plane % 8 == 0 && ((uintptr_t)W_planes & 15) == 0; }

// rows of fp32 values -> three planes [rows][K] of bf16 parts, K a multiple of 8
__global__ void __launch_bounds__(256) cut_rows_kernel(const float* __restrict__ src, int lda, int rows, int K, bf16* __restrict__ dst, int64_t plane) {
  pdl_launch();
  pdl_wait();
  const int per = K / 8;
  const int64_t n = (int64_t)rows * per;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const int64_t r = i / per;
    const int k = (int)(i - r * per) * 8;
    const float4* s = reinterpret_cast<const float4*>(src + r * lda + k);
    uint4 p1, p2, p3;
    cut8(s[0], s[1], p1, p2, p3);
    uint4* d = reinterpret_cast<uint4*>(dst + r * K + k);
    *d = p1;
    *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(d) + plane) = p2;
    *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(d) + 2 * plane) = p3;
  }
}
cudaError_t launch_cut_rows(const float* src, int lda, int rows, int K, void* dst, int64_t plane, cudaStream_t s) {
  if (K % 8 || lda % 4 || plane % 8 || (((uintptr_t)src | (uintptr_t)dst) & 15)) return cudaErrorInvalidValue;
  const int64_t n = (int64_t)rows * (K / 8);
  return launch_k(cut_rows_kernel, dim3((unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8)), dim3(256), 0, s, src, lda, rows, K, (bf16*)dst, plane);
}
