// Tensor-core projections for 9..128 activation rows (batched decode): y = x W^T with the roles
// of the MMA operands SWAPPED - a tile's 128-row operand is a block of WEIGHT rows and the batch
// is the N dimension (16 / 32 / 64 / 128 columns).  With the batch as the 128-row operand
// (gemm_tc.cu) every CTA re-reads the whole activation tile to stream only 32 weight rows; here a
// CTA streams 128 weight rows per 16-128 KB of activations, so shared-memory ingress is spent on
// the bytes that matter (weights are read exactly once from HBM, the HBM-bound regime of
// llama3.py:99-102,166-168,211 at small batch).  Matrices with few row blocks (QKV: 48, Wo / Wdown:
// 32 at D = 4096) are additionally split along K: every slice publishes its partial tile and the last
// one to arrive sums them in slice order (deterministic) before the fused epilogue.  The bf16-mode
// residual epilogue adds its slices into the residual stream with fp32 atomics instead (no reduction
// tail: 4 us per GEMM faster at the 8B shape); fp32 mode never reorders a sum.
//
// The accumulator is transposed (TMEM lane = output column n, TMEM column = activation row m), so
// the epilogue needs no shared-memory pass: for a fixed m the 32 lanes of a warp hold 32
// consecutive n - every global access is coalesced as it stands; RoPE / SwiGLU pairs are adjacent
// lanes (one shuffle).
#include <cuda.h>

#include <stdlib.h>
#include <algorithm>

#include "common.cuh"
#include "gemm_tc.h"

namespace {
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok, spins = 0;
  do {
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (!ok && ++spins > (1u << 26)) __trap();  // a protocol bug must fail the launch, not hang the GPU
  } while (!ok);
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(tm), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
// one lane of the (whole) warp, known as one to the compiler (see gemm_tc_dev.cuh)
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <int KIND>
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  if constexpr (KIND == TC_BF16) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
  } else {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
  }
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// 0 where not `on`: a predicate and no branch, so that a row of such loads is in flight together
__device__ __forceinline__ float ld_cluster_if(bool on, uint32_t a) {
  float v;
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\nmov.f32 %0, 0f00000000;\n@p ld.shared::cluster.f32 %0, [%1];\n}" : "=f"(v) : "r"(a), "r"((int)on) : "memory");
  return v;
}

constexpr int SW_THREADS = 224;  // warp 0 = weight copies, warp 1 = TMEM + MMA, warps 2-5 = epilogue, warp 6 = activation copies
// BNA = batch columns of the tile (activation rows padded up)
template <int KIND, int BNA> struct SwCfg {
  static constexpr int PARTS = KIND == TC_TF32X3 ? 2 : 1;
  static constexpr int BMW = 128;                       // weight rows of the MMA; a tile holds h <= BMW of them
  static constexpr int BK = KIND == TC_BF16 ? 64 : 32;  // elements per 128-byte row
  static constexpr int X_BYTES = BNA * 128;
  __host__ __device__ static constexpr int w_bytes(int h) { return (h + 7) / 8 * 1024; }
  __host__ __device__ static constexpr int stage_bytes(int h) { return PARTS * (w_bytes(h) + X_BYTES); }
  // (bf16 with four round-robin accumulators was measured: no gain at 8B batch 32, so one accumulator)
  static constexpr int NACC = KIND == TC_TF32X3 ? 4 : 1;
  static constexpr int AW = BNA < 32 ? 32 : BNA;        // TMEM columns from one accumulator to the next (read 32 at a time)
  static constexpr int CJ = BNA < 32 ? BNA : 32;        // rows of an epilogue chunk
  static constexpr int ACC_COLS = NACC * AW;
  static constexpr int NBUF = 2 * ACC_COLS <= 512 ? 2 : 1;
  static constexpr int TMEM_COLS = NBUF * ACC_COLS <= 32 ? 32 : NBUF * ACC_COLS <= 64 ? 64 : NBUF * ACC_COLS <= 128 ? 128
                                   : NBUF * ACC_COLS <= 256 ? 256 : 512;
  // The MMA reads BMW rows; behind a tile's h it reads whatever follows in shared memory (those accumulators are not looked at), so
  // low tiles leave room for more stages - what keeps DRAM busy is the bytes in flight - and the last stage is followed by a tile's rest.
  static constexpr int MAX_STAGES = 32, REST = BMW * 128, SMEM_MAX = 232448, BARS = 1024;
  __host__ __device__ static constexpr int stages(int h) {
    const int n = (SMEM_MAX - 1024 - BARS - REST) / stage_bytes(h);
    return n > MAX_STAGES ? MAX_STAGES : n;
  }
  static constexpr uint32_t FMT = KIND == TC_BF16 ? 1u : 2u;
  // D fp32, both operands K-major, N = BNA, M = 128
  static constexpr uint32_t IDESC = (1u << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(BNA >> 3) << 17) | ((128u >> 4) << 24);
};

// CL: the slices of a tile are a cluster, one item per CTA.  EPI_GATED: EPI_SWIGLU with any activation, with routing weights or without; the
// plain silu is EPI_SWIGLU.  Both are kernels of their own: as arguments their row bounds, branches and loops cost every other launch 0.1 -
// 0.5 us (9 rows, 2048 x 2048 added in place 3.89 : 4.16, 16384 x 2048 gated 13.3 : 13.8).
constexpr int EPI_GATED = 8;
template <int KIND, int BNA, int EPI, bool CL>
__global__ void __launch_bounds__(SW_THREADS, 1)
gemm_swap_kernel(const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                 const __grid_constant__ CUtensorMap tmX0, const __grid_constant__ CUtensorMap tmX1,
                 int rows, int N, int K, int h, int nst, int ksplit, float* part, int* tile_cnt, EpiArgs e) {
  using Cf = SwCfg<KIND, BNA>;
  using KVT = typename std::conditional<KIND == TC_BF16, bf16, float>::type;
  constexpr int PARTS = Cf::PARTS, NBUF = Cf::NBUF, CJ = Cf::CJ;
  const int W_BYTES = Cf::w_bytes(h), STAGE_BYTES = Cf::stage_bytes(h);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;
  const uint32_t bars = tiles + nst * STAGE_BYTES + Cf::REST;
  const uint32_t full0 = bars, empty0 = bars + 8 * nst, accfull0 = bars + 16 * nst, accempty0 = accfull0 + 16,
                 tmem_slot = accempty0 + 16;
  uint32_t* tmem_slot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tmem_slot - raw));

  const int warp = __shfl_sync(L3_FULL, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int tiles_w = (N + h - 1) / h;
  const int ntiles = tiles_w * ksplit;
  const int nkb = (K + Cf::BK - 1) / Cf::BK;
  const int kb_per = (nkb + ksplit - 1) / ksplit;
  auto tile_of = [&](int t) { return CL ? t / ksplit : t % tiles_w; };
  auto slice_of = [&](int t) { return CL ? t % ksplit : t / tiles_w; };
  pdl_launch();

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmW0));
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmX0));
    if (PARTS == 2) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmW1));
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmX1));
    }
    for (int s = 0; s < nst; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(accfull0 + 8 * b, 1); mbar_init(accempty0 + 8 * b, 4); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "n"(Cf::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // the copies' warp, which made the barriers, goes ahead of the TMEM allocation
  uint32_t tmem_base = 0;
  if (warp == 0) {
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"n"(SW_THREADS) : "memory");
  } else {
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(SW_THREADS) : "memory");
    tc_fence_after();
    tmem_base = *tmem_slot_ptr;
  }

  // The issuing warps run their loops whole, one elected lane issues, ring positions are counted: as one lane of a divergent warp with
  // two divisions per k-block the issue code took ~600 cycles per 16 KB of weights - 5.2 TB/s over the chip.  With that, with the gated
  // epilogue's values taken in front of its stores 32 x 28672 x 4096 went from 59.1 to 45.8 us, launched in a
  // row over weights that no cache holds (a plain read of them: 38.4).
  if (warp == 0 || warp == 6) {  // ---------------- copies: weights, activations
    // weights do not depend on the previous kernel: their first stages are requested before the
    // dependency wait; the activation boxes follow once the producer kernel's writes are visible
    if (warp == 6) pdl_wait();
    int s = 0;
    uint32_t ph = 1;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
      const int n0 = tile_of(t) * h, ks = slice_of(t);
      const int kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(empty0 + 8 * s, ph);
        const uint32_t st = tiles + s * STAGE_BYTES, bar = full0 + 8 * s;
        if (elect_one()) {
          if (warp == 0) {
            mbar_expect_tx(bar, PARTS * (h * 128 + Cf::X_BYTES));
            tma_load_2d(st, &tmW0, kb * Cf::BK, n0, bar);
            if (PARTS == 2) tma_load_2d(st + W_BYTES, &tmW1, kb * Cf::BK, n0, bar);
          } else {
            tma_load_2d(st + PARTS * W_BYTES, &tmX0, kb * Cf::BK, 0, bar);
            if (PARTS == 2) tma_load_2d(st + PARTS * W_BYTES + Cf::X_BYTES, &tmX1, kb * Cf::BK, 0, bar);
          }
        }
        __syncwarp();
        if (++s == nst) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {  // ---------------- MMA issuer
    int s = 0;
    uint32_t ph = 0, ti = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++ti) {
      const int ks = slice_of(t);
      const int kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      const uint32_t buf = ti % NBUF, use = ti / NBUF;
      if (use > 0) {
        mbar_wait(accempty0 + 8 * buf, (use - 1) & 1);
        tc_fence_after();
      }
      const uint32_t acc = tmem_base + buf * Cf::ACC_COLS;
      int third = 0;  // main accumulator of the next K slice (3xTF32)
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(full0 + 8 * s, ph);
        tc_fence_after();
        const uint32_t st = tiles + s * STAGE_BYTES;
        const uint64_t w_hi = umma_desc_sw128(st), x_hi = umma_desc_sw128(st + PARTS * W_BYTES);
        if (elect_one()) {
          const uint32_t more = kb > kb0;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint64_t adv = (uint64_t)(kk * 2);
            if (PARTS == 2) {
              const uint64_t w_lo = umma_desc_sw128(st + W_BYTES);
              const uint64_t x_lo = umma_desc_sw128(st + PARTS * W_BYTES + Cf::X_BYTES);
              int main = third + kk;
              while (main >= 3) main -= 3;
              const uint32_t corr = acc + 3 * Cf::AW, mainacc = acc + main * Cf::AW;
              tc_mma<KIND>(corr, w_lo + adv, x_hi + adv, Cf::IDESC, kk ? 1u : more);
              tc_mma<KIND>(corr, w_hi + adv, x_lo + adv, Cf::IDESC, 1u);
              tc_mma<KIND>(mainacc, w_hi + adv, x_hi + adv, Cf::IDESC, kk >= 3 ? 1u : more);
            } else {
              tc_mma<KIND>(acc, w_hi + adv, x_hi + adv, Cf::IDESC, kk ? 1u : more);
            }
          }
          tc_commit(empty0 + 8 * s);
          if (kb == kb1 - 1) tc_commit(accfull0 + 8 * buf);
        }
        __syncwarp();
        if (PARTS == 2) { third += 4; while (third >= 3) third -= 3; }
        if (++s == nst) { s = 0; ph ^= 1; }
      }
      if (kb0 >= kb1 && elect_one()) tc_commit(accfull0 + 8 * buf);  // a slice without blocks
      __syncwarp();
    }
  } else {  // ---------------- epilogue (warps 2-5): lane = output column, TMEM column = activation row
    pdl_wait();  // residual / position reads below depend on the previous kernel
    const int quarter = warp & 3;
    const int start_pos = (EPI == EPI_ROPE_KV) ? *e.pos_ptr : 0;
    uint32_t ti = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++ti) {
      const int n0 = tile_of(t) * h, ks = slice_of(t);
      const int kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      const uint32_t buf = ti % NBUF, use = ti / NBUF;
      mbar_wait(accfull0 + 8 * buf, use & 1);
      tc_fence_after();
      const uint32_t acc = tmem_base + buf * Cf::ACC_COLS + ((uint32_t)(quarter * 32) << 16);
      const int n = n0 + quarter * 32 + lane;       // this lane's output column
      const bool n_ok = quarter * 32 + lane < h && n < N && kb0 < kb1;
      const bool live = quarter * 32 < h && n0 + quarter * 32 < N && kb0 < kb1;  // warp-uniform
      auto load_acc = [&](int c0, float (&v)[32]) {
        tmem_ld32(acc + (uint32_t)c0, v);
        if (Cf::NACC == 4) {
          float w[32];
#pragma unroll
          for (int k2 = 1; k2 < 4; ++k2) {
            tmem_ld32(acc + (uint32_t)c0 + k2 * Cf::AW, w);
#pragma unroll
            for (int j = 0; j < CJ; ++j) v[j] += w[j];
          }
        }
      };
      const int Np = tiles_w * Cf::BMW;  // padded width of the K-split scratch [ksplit][BNA][Np]
      const int tw = tile_of(t), np = tw * Cf::BMW + quarter * 32 + lane;
      const bool det = CL || (ksplit > 1 && part != nullptr);  // else (residual epilogue only): fp32 atomics
      int m_lo = 0, m_hi = rows;  // rows that this CTA finishes
      float* mine = reinterpret_cast<float*>(smem_raw + (tiles - raw)) + quarter * 32 + lane;  // CL: [row][128 columns]
      if constexpr (CL) {
        // The slices' sums stay in shared memory - the ring, which nothing reads any more - and every CTA of the cluster adds up and
        // finishes its share of the rows, slices in order: the sums of the published form below without its trip through L2 and
        // without a last arriver that works alone.  40 greedy tokens of 32 sequences at the 8B shape 11120 -> 10960 us.
#pragma unroll 1
        for (int c0 = 0; c0 < BNA; c0 += 32) {
          if (c0 >= rows || !live) break;
          float v[32];
          load_acc(c0, v);
#pragma unroll
          for (int j = 0; j < CJ; ++j)
            if (c0 + j < rows) mine[(c0 + j) * Cf::BMW] = v[j];
        }
        __syncwarp();
        cluster_sync_all();
        m_lo = rows * ks / ksplit;
        m_hi = rows * (ks + 1) / ksplit;
      } else if (det) {
        // K-split: publish this slice's partial tile (for a fixed row the warp's 32 lanes store 32 consecutive
        // columns); the LAST slice of an output tile to arrive sums all slices in slice order - a fixed order,
        // so the result does not depend on timing - and runs the fused epilogue on the sum.
#pragma unroll 1
        for (int c0 = 0; c0 < BNA; c0 += 32) {
          if (c0 >= rows || !live) break;
          float v[32];
          load_acc(c0, v);
#pragma unroll
          for (int j = 0; j < CJ; ++j)
            if (c0 + j < rows) __stcg(part + ((size_t)ks * BNA + c0 + j) * Np + np, v[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(accempty0 + 8 * buf);
        // release: the CTA barrier orders the four warps' partial stores before thread 64's acq_rel atomic
        // (cumulative), whose acquire side + the next barrier order the last arriver's reads after all slices'
        asm volatile("bar.sync 2, 128;" ::: "memory");  // the four epilogue warps
        int* flag = reinterpret_cast<int*>(smem_raw + (tmem_slot - raw)) + 1;
        if (threadIdx.x == 64) {
          int old;
          asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(tile_cnt + tw) : "memory");
          *flag = (old == ksplit - 1);
          if (old == ksplit - 1) tile_cnt[tw] = 0;  // ready for the next launch
        }
        asm volatile("bar.sync 2, 128;" ::: "memory");
        const bool is_last = *flag != 0;
        asm volatile("bar.sync 2, 128;" ::: "memory");  // everyone has read the flag before it is reused
        if (!is_last) continue;
      }
#pragma unroll 1
      for (int c0 = m_lo; c0 < BNA; c0 += CJ) {
        if (c0 >= m_hi || !live) break;  // warp-uniform
        float v[32];
        if (CL) {
#pragma unroll
          for (int j = 0; j < CJ; ++j) v[j] = 0.f;
          for (int k2 = 0; k2 < ksplit; ++k2) {
            const uint32_t src = cluster_at(smem_u32(mine + c0 * Cf::BMW), (uint32_t)k2);
            float w[32];
#pragma unroll
            for (int j = 0; j < CJ; ++j) w[j] = ld_cluster_if(c0 + j < m_hi, src + j * Cf::BMW * 4);
#pragma unroll
            for (int j = 0; j < CJ; ++j) v[j] += w[j];
          }
        } else if (!det) {
          load_acc(c0, v);
          if (c0 + 32 >= BNA || c0 + 32 >= rows) {  // last TMEM read of this tile: hand the buffer back early
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty0 + 8 * buf);
          }
        } else {  // sum of the slices' partials, slice 0 first
#pragma unroll
          for (int j = 0; j < CJ; ++j) v[j] = 0.f;
          // unconditional loads (the scratch holds BNA rows per slice): all 32 are in flight before the first add -
          // guarded ones are issued three at a time, ~10 dependent L2 round trips per slice
          for (int k2 = 0; k2 < ksplit; ++k2) {
            const float* src = part + ((size_t)k2 * BNA + c0) * Np + np;
            float w[32];
#pragma unroll
            for (int j = 0; j < CJ; ++j) w[j] = __ldcg(src + (size_t)j * Np);
#pragma unroll
            for (int j = 0; j < CJ; ++j) v[j] += w[j];
          }
        }
        if constexpr (EPI == EPI_STORE) {
          if (e.unary) {
#pragma unroll
            for (int j = 0; j < CJ; ++j) v[j] = unary_act(e.unary, v[j]);
          }
#pragma unroll
          for (int j = 0; j < CJ; ++j) {
            const int m = c0 + j;
            if (m < m_hi && n_ok) {
              const size_t o = (size_t)m * e.ld_out + n;
              if (e.out_lo) { float hi, lo; split_tf32(v[j], hi, lo); e.out[o] = hi; e.out_lo[o] = lo; }
              else if (e.out) e.out[o] = v[j];
              if (e.out_bf16) e.out_bf16[o] = __float2bfloat16_rn(v[j]);
            }
          }
        } else if constexpr (EPI == EPI_RESID) {
          if (ksplit == 1 || det) {
            // clamped instead of guarded, so that all 32 loads are in flight together (values of clamped
            // duplicates are not used)
            const int nc = min(n, N - 1);
            float rr[32];
#pragma unroll
            for (int j = 0; j < CJ; ++j) rr[j] = e.resid[(size_t)min(c0 + j, rows - 1) * e.ld_out + nc];
#pragma unroll
            for (int j = 0; j < CJ; ++j)
              if (c0 + j < m_hi && n_ok) e.out[(size_t)(c0 + j) * e.ld_out + n] = rr[j] + v[j];
          } else {  // bf16 mode: the slices add their partials into the residual stream in place (out == resid)
#pragma unroll
            for (int j = 0; j < CJ; ++j)
              if (c0 + j < rows && n_ok) atomicAdd(e.out + (size_t)(c0 + j) * e.ld_out + n, v[j]);
          }
        } else if constexpr (EPI == EPI_SWIGLU || EPI == EPI_GATED) {
          // weight rows interleave gate_j, up_j: an even lane holds the gate, its odd neighbour the up value.  The even lane takes the
          // chunk's first half of the rows, the odd one the second; all values before the first store, the activation decided once.
          // silu with expf and a full reciprocal, in both modes: the fast forms take 0.7 us less at 32 x 28672 x 4096 and 3.5 us at 100 rows
          // but lose bits of every value, and all of them from -87.4 down.
          constexpr int HF = CJ / 2;
          const bool odd = lane & 1;
          const int mb = c0 + (odd ? HF : 0);
          float gt[HF], hv[HF];
#pragma unroll
          for (int j = 0; j < HF; ++j) {
            const float got = __shfl_xor_sync(L3_FULL, odd ? v[j] : v[j + HF], 1);
            gt[j] = odd ? got : v[j];
            hv[j] = odd ? v[j + HF] : got;
          }
          if (EPI == EPI_SWIGLU || (e.act == GLU_SILU && !e.glu_w)) {
#pragma unroll
            for (int j = 0; j < HF; ++j) hv[j] = silu_ref(gt[j]) * hv[j];
          } else if (e.act == GLU_GELU_TANH && !e.glu_w) {
#pragma unroll
            for (int j = 0; j < HF; ++j) hv[j] = gelu_tanh_ref(gt[j]) * hv[j];
          } else if (e.act == GLU_CLAMP && !e.glu_w) {
            const float limit = e.act_limit, slope = e.act_slope;
#pragma unroll
            for (int j = 0; j < HF; ++j) hv[j] = glu_clamp<KIND == TC_BF16>(limit, slope, gt[j], hv[j]);
          } else {
#pragma unroll
            for (int j = 0; j < HF; ++j) {
              const float w = e.glu_w && mb + j < rows && n_ok ? glu_in_weight(e, mb + j, n >> 1) : 1.f;
              hv[j] = glu_pair<KIND == TC_BF16>(e, gt[j] * w, hv[j] * w);
            }
          }
          if (n_ok) {
            const size_t o = (size_t)mb * e.ld_out + (n >> 1);
#pragma unroll
            for (int j = 0; j < HF; ++j)
              if (mb + j < m_hi) {
                const size_t oj = o + (size_t)j * e.ld_out;
                if (e.out_lo) split_tf32(hv[j], e.out[oj], e.out_lo[oj]);
                else if (e.out) e.out[oj] = hv[j];
                if (e.out_bf16) e.out_bf16[oj] = __float2bfloat16_rn(hv[j]);
              }
          }
        } else if constexpr (EPI == EPI_ROPE_KV) {
          const int qcols = e.HN * e.HD, kcols = e.KVHN * e.HD;
          const bool is_q = n < qcols, is_k = !is_q && n < qcols + kcols;
          const int within = is_q ? n : (is_k ? n - qcols : n - qcols - kcols);
          const int hh = within / e.HD, d = within % e.HD;
          // lane l looks up row c0 + l - sequence, position, its row of the cache (-1: padding) - and the others ask it: a division and
          // its loads per lane instead of 64 divisions and, in the store loop, a length's load per row (no load may move above a
          // store that could alias it).  Table entries of all 32 rows come ahead of the stores as well.  32 x 6144 x 4096: 25.7 -> 19.5 us
          const int lm = min(c0 + lane, rows - 1), lb = lm / e.L, lt = lm - lb * e.L;  // clamped: rows past the end are not used
          const int lpos = (e.row_pos ? __ldg(e.row_pos + lb) : start_pos) + lt;
          const int lrow = !e.row_len || lt < __ldg(e.row_len + lb) ? lb * e.KVHN * e.M + lpos : -1;
          float cs[32], sn[32];
#pragma unroll
          for (int j = 0; j < CJ; ++j) {
            const size_t ti = (size_t)__shfl_sync(L3_FULL, lpos, j) * (e.HD >> 1) + (d >> 1);
            cs[j] = (is_q || is_k) ? __ldg(e.cos_tab + ti) : 1.f;
            sn[j] = (is_q || is_k) ? __ldg(e.sin_tab + ti) : 0.f;
          }
#pragma unroll
          for (int j = 0; j < CJ; ++j) {
            const float other = __shfl_xor_sync(L3_FULL, v[j], 1);  // the pair's partner (llama3.py:41-76)
            const int m = c0 + j, row = __shfl_sync(L3_FULL, lrow, j);
            if (m >= m_hi || !n_ok) continue;
            float r = v[j];
            // even: x0 c - x1 s, odd: x0 s + x1 c
            if (is_q || is_k) r = (lane & 1) ? other * sn[j] + v[j] * cs[j] : v[j] * cs[j] - other * sn[j];
            if (is_q) {
              const size_t o = (size_t)m * e.ld_out + n;
              if (e.out) e.out[o] = r;
              if (e.out_bf16) e.out_bf16[o] = __float2bfloat16_rn(r);
            } else if (row >= 0) {
              KVT* c = (KVT*)(is_k ? e.cache_k : e.cache_v) + ((size_t)row + (size_t)hh * e.M) * e.HD + d;
              *c = from_f32<KVT>(r);
            }
          }
        } else {  // EPI_ARGMAX (llama3.py:320): per activation row, the warp's best (value, first index)
          // two warp-wide integer reductions per row (redux.sync) on the order-preserving key halves:
          // the largest value first, then the smallest column among the lanes that hold it
#pragma unroll
          for (int j = 0; j < CJ; ++j) {
            const int m = c0 + j;
            if (m >= m_hi) continue;  // warp-uniform
            uint32_t kv = 0u;  // ordered bits of the value; 0 = no candidate
            if (n_ok) {
              const uint32_t b = __float_as_uint(v[j]);
              kv = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
            }
            const uint32_t best_v = __reduce_max_sync(L3_FULL, kv);
            const uint32_t best_n = __reduce_min_sync(L3_FULL, (n_ok && kv == best_v) ? (uint32_t)n : 0xffffffffu);
            if (lane == 0 && best_n != 0xffffffffu)
              atomicMax(e.best + m, ((unsigned long long)best_v << 32) | (unsigned long long)(0xffffffffu - (uint32_t)(e.col_offset + (int)best_n)));
          }
        }
      }
      if (!det && !live) {  // nothing was read: still hand the buffer back
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(accempty0 + 8 * buf);
      }
    }
  }
  if constexpr (CL) {
    if (warp < 2 || warp == 6) cluster_sync_all();  // the others have met where the slices' sums were complete
    cluster_sync_all();                             // nobody leaves while its sums are read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(Cf::TMEM_COLS));
  }
}

int sm_count() {
  static int n[16] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!n[dev & 15]) cudaDeviceGetAttribute(&n[dev & 15], cudaDevAttrMultiProcessorCount, dev);
  return n[dev & 15] > 0 ? n[dev & 15] : 148;
}

template <int KIND, int BNA, int EPI, bool CL>
cudaError_t launch_sw_t(const TcGemmArgs& a, cudaStream_t s) {
  using Cf = SwCfg<KIND, BNA>;
  auto kern = gemm_swap_kernel<KIND, BNA, EPI, CL>;
  static bool attr_done[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_done[dev & 15]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cf::SMEM_MAX);
    if (e != cudaSuccess) return e;
    attr_done[dev & 15] = true;
  }
  const bool b16 = KIND == TC_BF16;
  const int h = a.bn;
  const CUtensorMap* W0 = tc_get_map(a.W[0], b16, a.N, a.K, h);
  const CUtensorMap* X0 = tc_get_map(a.A[0], b16, a.rows, a.K, BNA);
  const CUtensorMap* W1 = Cf::PARTS == 2 ? tc_get_map(a.W[1], b16, a.N, a.K, h) : W0;
  const CUtensorMap* X1 = Cf::PARTS == 2 ? tc_get_map(a.A[1], b16, a.rows, a.K, BNA) : X0;
  if (!W0 || !X0 || !W1 || !X1) return cudaErrorInvalidValue;
  dim3 grid(std::min((a.N + h - 1) / h * a.ksplit, sm_count()));
  // no more stages than a CTA has k-blocks
  const int nkb = (a.K + Cf::BK - 1) / Cf::BK, items = ((a.N + h - 1) / h * a.ksplit + (int)grid.x - 1) / (int)grid.x;
  const int nst = std::max(2, std::min(Cf::stages(h), (nkb + a.ksplit - 1) / a.ksplit * items));
  if (CL && a.rows * Cf::BMW * 4 > nst * Cf::stage_bytes(h)) return cudaErrorInvalidValue;  // the sums lie in the ring: four blocks and more
  if (CL) grid.x = (a.N + h - 1) / h * a.ksplit;
  return launch_kc(kern, grid, dim3(SW_THREADS), (size_t)(nst * Cf::stage_bytes(h) + Cf::REST + 1024 + Cf::BARS), s, CL ? a.ksplit : 1, *W0, *W1, *X0, *X1, a.rows, a.N, a.K, h, nst, a.ksplit, a.part, a.tile_cnt, a.e);
}

template <int KIND, int BNA, bool CL>
cudaError_t launch_sw_e(const TcGemmArgs& a, cudaStream_t s) {
  switch (a.epi) {
    case EPI_STORE: return launch_sw_t<KIND, BNA, EPI_STORE, CL>(a, s);
    case EPI_RESID: return launch_sw_t<KIND, BNA, EPI_RESID, CL>(a, s);
    case EPI_SWIGLU:
      return a.e.act == GLU_SILU && !a.e.glu_w ? launch_sw_t<KIND, BNA, EPI_SWIGLU, CL>(a, s) : launch_sw_t<KIND, BNA, EPI_GATED, CL>(a, s);
    case EPI_ARGMAX: return launch_sw_t<KIND, BNA, EPI_ARGMAX, CL>(a, s);
    default: return launch_sw_t<KIND, BNA, EPI_ROPE_KV, CL>(a, s);
  }
}
template <int KIND, int BNA>
cudaError_t launch_sw_c(const TcGemmArgs& a, bool cluster, cudaStream_t s) {
  return cluster ? launch_sw_e<KIND, BNA, true>(a, s) : launch_sw_e<KIND, BNA, false>(a, s);
}
}  // namespace

bool gemm_swap_supported(int rows, int N) { return rows >= 1 && rows <= 128 && N >= 128; }

// bf16 mode's residual epilogue may add its slices in place, in any order (fp32 mode must not reorder a sum).  Results then differ from
// run to run in their last bits, so that is kept to products that are long (at least 16 k-blocks; shorter ones take less than 8000
// cycles whole) and leave more than half of the SMs without a row block; the others are summed in slice order, or not cut.
static bool adds_in_place(const TcGemmArgs& a, int sms) {
  static const int resid_atomic = [] { const char* v = getenv("L3_SWAP_RESID_ATOMIC"); return v ? atoi(v) : 1; }();
  return a.epi == EPI_RESID && a.kind == TC_BF16 && a.e.out == a.e.resid && resid_atomic && (a.K + 63) / 64 >= 16 && (a.N + 127) / 128 * 2 <= sms;
}
// Clusters of n CTAs with all of an SM's shared memory each that the device holds at once, whatever its GPCs' populations: eight of them with even
// numbers of SMs, of which each leaves up to n - 1 (n - 2 for even n) without a cluster.  148 SMs, n = 2 .. 8: 74, 44, 33, 24, 20, 15, 13
// (cudaOccupancyMaxActiveClusters there: 74, 45, 33, 26, 22, 15, 15).  By the SM count alone, so that one product is cut, and its sums come,
// alike on every device of that count.
static int clusters_of(int n, int sms) { return std::max(0, (sms - 8 * (n - 1 & ~1) + n - 1) / n); }
// Tile height and K split, by the cycles of the busiest CTA: a k-block takes the issue loops ~500 cycles (fp32 mode, two parts and three
// products: 750 - 980 with the columns), or its share of DRAM (3560 bytes per cycle for all CTAs that stream).  Slices that are added in place
// cost little (9 x 2048 x 4096, 1, 2, 4, 8 slices 18.0, 12.4, 10.1, 8.6 us); a cluster's, taken where all tiles' clusters are resident at once,
// 3000 cycles whatever their number (with 1800, as one would count from the kernel alone, short products are cut that run faster whole under
// their neighbours' tails: 28 x 7680 x 760 6.7 : 7.8 us); published and summed ones 2800 and more with each slice and row (9 x 6144 x 4096 two
// slices as clusters 13.0 us, three published 11.6).  More tiles than SMs: the height that makes the last round full (28672 rows: 293 tiles of
// 98 instead of 224 of 128 - 100 rows 57.5 -> 56.2 us).  Over 547 shapes in both modes (profiles/gemm_swap_cuts.jsonl) the choice is 1 % behind
// the best of all cuts in the mean and takes 0.83 of the time of the plan and kernel without clusters.
static void pick_swap(const TcGemmArgs& a, int bna, int sms, int* h_out, int* ks_out, bool* cl_out) {
  static const int max_split = [] { const char* v = getenv("L3_SWAP_KSPLIT"); return v ? atoi(v) : 8; }();
  static const int det_epi = [] { const char* v = getenv("L3_SWAP_KSPLIT_DET"); return v ? atoi(v) : 1; }();
  const bool b16 = a.kind == TC_BF16, atomic = adds_in_place(a, sms);
  const int parts = b16 ? 1 : 2, nkb = (a.K + (b16 ? 63 : 31)) / (b16 ? 64 : 32);
  const int rounds = ((a.N + 127) / 128 + sms - 1) / sms;
  int h = 128;
  if (rounds > 1) h = std::min(128, ((a.N + sms * rounds - 1) / (sms * rounds) + 1) & ~1);
  const int tiles = (a.N + h - 1) / h;
  double best = 0;
  *cl_out = false;
  for (int ks = 1; ks <= std::max(1, atomic ? 8 : std::min(8, max_split)); ++ks) {
    const int per = (nkb + ks - 1) / ks;
    if (ks > 1 && (per < 4 || (ks - 1) * per >= nkb)) break;
    const bool cl = ks > 1 && !atomic && det_epi && clusters_of(ks, sms) >= tiles;
    if (ks > 1 && !atomic && !cl && (!a.part || !a.tile_cnt || tiles > a.tile_cnt_len || (size_t)bna * tiles * 128 * sizeof(float) * ks > a.part_bytes ||
                              !(det_epi || a.epi == EPI_RESID))) break;
    const double issue = b16 ? 500 : 720 + 2.0 * bna, slice = 22.0 * bna + (b16 ? 0 : 8.0 * a.rows);
    const int full = tiles * ks / sms, rest = tiles * ks % sms;
    double c = full * per * std::max(issue, h * 128.0 * parts * sms / 3560);
    if (rest) c += per * std::max(issue, h * 128.0 * parts * rest / 3560);
    if (ks > 1) c += atomic ? 380 + 2.0 * ks * bna : cl ? 3000 : 2800 + slice * ks;
    if (best == 0 || c < best) { best = c; *ks_out = ks; *cl_out = cl; }
  }
  *h_out = h;
}

static int batch_cols(int rows) { return rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128; }
TcPlan gemm_swap_plan(const TcGemmArgs& a) {
  const int sms = sm_count();
  TcPlan p{1, 128, 1, 0};
  pick_swap(a, batch_cols(a.rows), sms, &p.width, &p.slices, &p.cluster);
  p.any_order = p.slices > 1 && adds_in_place(a, sms);
  return p;
}

cudaError_t launch_gemm_swap(const TcGemmArgs& args, cudaStream_t s) {
  TcGemmArgs a = args;
  const int bna = batch_cols(a.rows);
  TcPlan p = gemm_swap_plan(a);
  if (a.no_cluster) {
    if (!a.part || !a.tile_cnt) return cudaErrorInvalidValue;
    p.cluster = false;
  }
  a.bn = p.width; a.ksplit = p.slices;
  if (p.any_order) a.part = nullptr;
  // Measured and rejected at the 8B shape, batch 32 (profiles/swap_gemm_experiments.txt): a tile-contiguous copy of the weights read
  // with one 16 KB bulk copy per stage (not DRAM page locality), and the slices of a row block sharing its reduction + epilogue by rows
  // behind a cooperative launch (QKV 37 vs 29 us).  Later: tiles that start their turn over K one block apart (the activation boxes are
  // no hot spot), low tiles in place of a K split (42 rows x 147 CTAs for QKV: 17 vs 14 us, the issue loops' cycles per block remain).
  if (a.kind == TC_BF16) {
    switch (bna) {
      case 16: return launch_sw_c<TC_BF16, 16>(a, p.cluster, s);
      case 32: return launch_sw_c<TC_BF16, 32>(a, p.cluster, s);
      case 64: return launch_sw_c<TC_BF16, 64>(a, p.cluster, s);
      default: return launch_sw_c<TC_BF16, 128>(a, p.cluster, s);
    }
  }
  switch (bna) {
    case 16: return launch_sw_c<TC_TF32X3, 16>(a, p.cluster, s);
    case 32: return launch_sw_c<TC_TF32X3, 32>(a, p.cluster, s);
    case 64: return launch_sw_c<TC_TF32X3, 64>(a, p.cluster, s);
    default: return launch_sw_c<TC_TF32X3, 128>(a, p.cluster, s);
  }
}
