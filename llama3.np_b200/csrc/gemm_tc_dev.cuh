// Device side of the tcgen05 / TMA / TMEM GEMM (see gemm_tc.cu for the description): PTX wrappers, tile
// configuration and the warp-specialised pipeline as device functions.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "gemm_tc.h"

// debug timeline (l3_debug_tc_timeline): the first CTA stamps clock64 at pipeline milestones when it is given somewhere to
#define TC_STAMP(dbg, i)                                        \
  do {                                                          \
    if (dbg && blockIdx.x == 0) dbg[i] = clock64();             \
  } while (0)

// ------------------------------------------------------------------------------ PTX wrappers
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
// as above, but a wait that runs out sets *fail, and no wait of the CTA lasts from then on: the kernel runs to its end
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
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// between the two CTAs of a pair: an arrival and a tile load that complete at a shared::cluster address (cluster_at); products over both CTAs' operand tiles and the commit that reports them to both
__device__ __forceinline__ void pair_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(tm), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum) : "memory");
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
// 32 lanes x 32 consecutive fp32 columns -> 32 registers per thread (thread = TMEM lane)
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

// K-major, 128-byte-swizzled operand tile: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFF) >> 4)  // start address (16-byte units)
         | ((uint64_t)1 << 16)                   // leading byte offset (unused for swizzled K-major)
         | ((uint64_t)(1024 >> 4) << 32)         // stride byte offset: 8 rows x 128 B
         | ((uint64_t)1 << 46)                   // descriptor version (Blackwell)
         | ((uint64_t)2 << 61);                  // SWIZZLE_128B
}

// BN: columns of an output tile; 0 (bf16 only): any multiple of 32 up to 256, given at run time.  CG: CTAs that share a tile of
// CG * 128 rows - each loads its own 128 rows of A and its 1 / CG of the tile's weight rows, and the first one's products (cta_group::2)
// read both and leave every CTA its own rows' accumulators.
template <int KIND, int BN, int CG> struct TcCfg {
  static_assert(BN || KIND == TC_BF16, "widths at run time: bf16 only");
  static_assert(CG == 1 || BN == 0, "pairs of CTAs: widths at run time only");
  static constexpr int PARTS = KIND == TC_BF16 ? 1 : 2;
  static constexpr int BM = 128;
  static constexpr int BK = KIND == TC_BF16 ? 64 : 32;  // elements per 128-byte row
  static constexpr int A_BYTES = BM * 128;
  __host__ __device__ static constexpr int b_bytes(int bn) { return bn / CG * 128; }
  __host__ __device__ static constexpr int stage_bytes(int bn) { return PARTS * (A_BYTES + b_bytes(bn)); }
  static constexpr int NACC = KIND == TC_TF32X3 ? 4 : (KIND == TC_TF32X3_2 ? 2 : 1);  // main accumulators + 1 correction, or 1
  static constexpr int NMAIN = NACC > 1 ? NACC - 1 : 1;
  static constexpr int NBUF = 2 * NACC * BN <= 512 ? 2 : 1;  // double-buffered: epilogue(i) overlaps mainloop(i+1)
  __host__ __device__ static constexpr int tmem_cols(int bn) {
    return NBUF * NACC * bn <= 32 ? 32 : NBUF * NACC * bn <= 64 ? 64 : NBUF * NACC * bn <= 128 ? 128 : NBUF * NACC * bn <= 256 ? 256 : 512;
  }
  static constexpr int EPI_BYTES = 8 * 32 * 128;          // per epilogue warp a staging tile [32 rows][32 columns] fp32
  static constexpr int SMEM_MAX = 232448;
  __host__ __device__ static constexpr int stages(int bn) {
    const int n = (SMEM_MAX - 1024 - 512 - EPI_BYTES) / stage_bytes(bn);
    return n > 8 ? 8 : n;
  }
  __host__ __device__ static constexpr int smem(int bn, int nst) { return nst * stage_bytes(bn) + EPI_BYTES + 1024 /*align*/ + 512 /*barriers*/; }
  // instruction descriptor: D fp32, A/B bf16 or tf32, both K-major, N = bn, M = CG * 128
  static constexpr uint32_t FMT = KIND == TC_BF16 ? 1u : 2u;
  __host__ __device__ static constexpr uint32_t idesc(int bn) {
    return (1u << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(CG * 128 >> 4) << 24);
  }
};

// The pipeline state of one CTA: shared-memory ring + barriers, TMEM base
struct TcPipe {
  uint8_t* smem_raw;
  uint32_t raw, tiles, epi0, full0, empty0, accfull0, accempty0, peer, tmem_slot, tmem_base;
  int nst, bn, rank;
  volatile int* fail;  // set when a wait ran out
  unsigned long long* dbg;
};

// rows in groups (TcGemmArgs::groups)
struct TcGroups { const int* tiles; int n, k; };

// TC_THREADS: warp 0 = TMA, warp 1 = TMEM + MMA, warps 2-9 = epilogue.  smem: nst stages | EPI_BYTES | barriers.
// Only the barriers stand between a kernel's start and its first copy: TMEM is handed out meanwhile, and the warps that use it meet
// in tc_pipe_ready.
constexpr int TC_THREADS = 320;
template <int KIND, int BN, int CG>
__device__ __forceinline__ void tc_pipe_setup(TcPipe& p, uint8_t* smem_raw, int nst, int bn) {
  using Cf = TcCfg<KIND, BN, CG>;
  p.smem_raw = smem_raw;
  p.raw = smem_u32(smem_raw);
  p.tiles = (p.raw + 1023u) & ~1023u;
  p.nst = nst;
  p.bn = bn;
  p.rank = CG == 1 ? 0 : (int)(blockIdx.x % CG);  // clusters are CG consecutive blocks
  p.epi0 = p.tiles + nst * Cf::stage_bytes(bn);
  const uint32_t bars = p.epi0 + Cf::EPI_BYTES;  // full[nst] | empty[nst] | accfull[2] | accempty[2] | peer | tmem ptr | flag | fail
  p.full0 = bars; p.empty0 = bars + 8 * nst; p.accfull0 = bars + 16 * nst; p.accempty0 = p.accfull0 + 16;
  p.peer = p.accempty0 + 16;
  p.tmem_slot = p.peer + 8;
  p.fail = reinterpret_cast<volatile int*>(smem_raw + (p.tmem_slot - p.raw)) + 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < nst; ++s) { mbar_init(p.full0 + 8 * s, 1); mbar_init(p.empty0 + 8 * s, 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(p.accfull0 + 8 * b, 1); mbar_init(p.accempty0 + 8 * b, 8 * CG); }
    mbar_init(p.peer, 1);
    *p.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (CG == 2) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (CG == 1) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(p.tmem_slot), "r"(Cf::tmem_cols(bn)));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    } else {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(p.tmem_slot), "r"(Cf::tmem_cols(bn)));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
  }
  if (CG == 2) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // the other CTA's barriers stand before anything arrives there
    if (p.rank && warp == 1 && lane == 0) pair_arrive(cluster_at(p.peer, 0));  // this CTA's TMEM is there: the first one's products may write to it
  }
  __syncwarp();
}
// Barriers and TMEM are there for the products' warp and the epilogue's; the copies' warp, which made the barriers, goes ahead.
__device__ __forceinline__ void tc_pipe_ready(TcPipe& p) {
  if (threadIdx.x < 32) {
    asm volatile("bar.arrive 1, %0;" ::"n"(TC_THREADS) : "memory");
    return;
  }
  tc_fence_before();
  asm volatile("bar.sync 1, %0;" ::"n"(TC_THREADS) : "memory");
  tc_fence_after();
  p.tmem_base = *reinterpret_cast<uint32_t*>(p.smem_raw + (p.tmem_slot - p.raw));
}

template <int KIND, int BN, int CG>
__device__ __forceinline__ void tc_pipe_teardown(TcPipe& p, int* err) {
  using Cf = TcCfg<KIND, BN, CG>;
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *p.fail) {
    __nanosleep(1000000);  // copies still in flight land before the shared memory is given up
    if (!err) __trap();    // nobody to tell: the launch fails
    *err = 1;
  }
  __syncthreads();
  if (CG == 2) cluster_sync_all();  // nothing of the other CTA is under way to this one any more
  if ((threadIdx.x >> 5) == 1) {
    if constexpr (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(p.tmem_base), "r"(Cf::tmem_cols(p.bn)));
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(p.tmem_base), "r"(Cf::tmem_cols(p.bn)));
  }
}


// One GEMM over the tiles first_tile, first_tile + tile_stride, ...; returns when this warp's role is done
// (the epilogue warps: all their global stores issued).
template <int KIND, int BN, int CG, int EPI>
__device__ __forceinline__ void tc_gemm_run(TcPipe& p, const CUtensorMap* tmA0, const CUtensorMap* tmA1, const CUtensorMap* tmB0,
                                            const CUtensorMap* tmB1, int rows, int N, int K, int a_box_rows, int ksplit, float* part,
                                            int* tile_cnt, const TcGroups& grp, const EpiArgs& e, int first_tile, int tile_stride) {
  using Cf = TcCfg<KIND, BN, CG>;
  using KVT = typename std::conditional<KIND == TC_BF16, bf16, float>::type;
  constexpr int PARTS = Cf::PARTS, NBUF = Cf::NBUF;
  const int STAGES = p.nst, bn = BN ? BN : p.bn, rank = CG == 1 ? 0 : p.rank;
  const int B_BYTES = Cf::b_bytes(bn), STAGE_BYTES = Cf::stage_bytes(bn), ACC_COLS = Cf::NACC * bn;
  volatile int* const fail = p.fail;
  const uint32_t tiles = p.tiles, full0 = p.full0, empty0 = p.empty0, accfull0 = p.accfull0, accempty0 = p.accempty0;
  const int warp = __shfl_sync(L3_FULL, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  constexpr int TM = CG * Cf::BM;  // rows of an output tile
  const bool grouped = KIND == TC_BF16 && grp.tiles;
  const int tiles_m = grouped ? grp.tiles[0] : (rows + TM - 1) / TM, tiles_n = (N + bn - 1) / bn;
  const int ntiles_mn = tiles_m * tiles_n;
  const int ntiles = ntiles_mn * ksplit;  // K-split: tile t = (k slice t / ntiles_mn, output tile t % ntiles_mn)
  const int nkb = (K + Cf::BK - 1) / Cf::BK;
  const int kb_per = (nkb + ksplit - 1) / ksplit;

  // The two issuing warps walk their loops whole, one elected lane issues, and the ring position is counted, not divided for: with one
  // lane of a divergent warp and two divisions a k-block cost its issuers 730 cycles whatever the tile's width (products alone: 512 at
  // 256 columns, 256 at 128; copies alone 600 -> 450).
  if (warp == 0) {  // ---------------- TMA producer
    int s = 0;
    uint32_t ph = 1;
    for (int t = first_tile; t < ntiles; t += tile_stride) {
      const int tmn = t % ntiles_mn, ks = t / ntiles_mn;
      const int g = grouped ? grp.tiles[1 + tmn % tiles_m] : 0, kg = g * grp.k;
      const int m0 = (tmn % tiles_m) * TM + rank * Cf::BM, n0 = (tmn / tiles_m) * bn + rank * (bn / CG) + g * grp.n;
      const int kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(empty0 + 8 * s, ph, fail);
        const uint32_t st = tiles + s * STAGE_BYTES;
        if (elect_one()) {
          if constexpr (CG == 2) {  // both CTAs' tiles are counted by the first one's barrier, where the products wait for them
            const uint32_t bar = cluster_at(full0 + 8 * s, 0);
            if (rank == 0) mbar_expect_tx(full0 + 8 * s, CG * STAGE_BYTES);
            pair_load_2d(st, tmA0, kb * Cf::BK, m0, bar);
            pair_load_2d(st + Cf::A_BYTES, tmB0, kb * Cf::BK + kg, n0, bar);
          } else {
            // the A box holds only the rows that exist (decode batches of 9..127 rows): rows beyond it
            // keep stale shared memory, which only feeds accumulator rows the epilogue never reads
            mbar_expect_tx(full0 + 8 * s, PARTS * (a_box_rows * 128 + B_BYTES));
            tma_load_2d(st, tmA0, kb * Cf::BK, m0, full0 + 8 * s);
            tma_load_2d(st + PARTS * Cf::A_BYTES, tmB0, kb * Cf::BK + kg, n0, full0 + 8 * s);
            if (PARTS == 2) {
              tma_load_2d(st + Cf::A_BYTES, tmA1, kb * Cf::BK, m0, full0 + 8 * s);
              tma_load_2d(st + PARTS * Cf::A_BYTES + B_BYTES, tmB1, kb * Cf::BK, n0, full0 + 8 * s);
            }
          }
          if (t == first_tile && kb - kb0 < 12) TC_STAMP(p.dbg, 2 + kb - kb0);
        }
        __syncwarp();
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {  // ---------------- MMA issuer (of a pair: its first CTA's)
      if (CG == 2) mbar_wait(p.peer, 0, fail);
      int s = 0;
      uint32_t ph = 0, ti = 0;
      const uint32_t idesc = Cf::idesc(bn);
      for (int t = first_tile; t < ntiles; t += tile_stride, ++ti) {
        const uint32_t buf = ti % NBUF, use = ti / NBUF;
        if (use > 0) {  // the epilogue must have drained this accumulator buffer
          mbar_wait(accempty0 + 8 * buf, (use - 1) & 1, fail);
          tc_fence_after();
        }
        const uint32_t acc = p.tmem_base + buf * ACC_COLS;
        const int ks = t / ntiles_mn;
        const int kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
        int third = 0;  // main accumulator of the next K slice (3xTF32)
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(full0 + 8 * s, ph, fail);
          tc_fence_after();
          const uint32_t st = tiles + s * STAGE_BYTES;
          const uint64_t a_hi = umma_desc_sw128(st), b_hi = umma_desc_sw128(st + PARTS * Cf::A_BYTES);
          if (elect_one()) {
            if (ti == 0 && kb - kb0 < 12) TC_STAMP(p.dbg, 16 + kb - kb0);
            const uint32_t more = kb > kb0;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {  // 4 slices of 32 bytes along K inside the swizzle atom
              const uint64_t adv = (uint64_t)(kk * 2);
              if constexpr (PARTS == 2) {
                const uint64_t a_lo = umma_desc_sw128(st + Cf::A_BYTES);
                const uint64_t b_lo = umma_desc_sw128(st + PARTS * Cf::A_BYTES + B_BYTES);
                int main = third + kk;
                while (main >= Cf::NMAIN) main -= Cf::NMAIN;
                const uint32_t corr = acc + Cf::NMAIN * bn, mainacc = acc + main * bn;
                tc_mma<KIND>(corr, a_lo + adv, b_hi + adv, idesc, kk ? 1u : more);
                tc_mma<KIND>(corr, a_hi + adv, b_lo + adv, idesc, 1u);
                tc_mma<KIND>(mainacc, a_hi + adv, b_hi + adv, idesc, kk >= Cf::NMAIN ? 1u : more);
              } else if constexpr (CG == 2) {
                pair_mma(acc, a_hi + adv, b_hi + adv, idesc, kk ? 1u : more);
              } else {
                tc_mma<KIND>(acc, a_hi + adv, b_hi + adv, idesc, kk ? 1u : more);
              }
            }
            // frees the stage once these MMAs have read it; behind the last block: the accumulator is complete
            if constexpr (CG == 2) {
              pair_commit(empty0 + 8 * s);
              if (kb == kb1 - 1) pair_commit(accfull0 + 8 * buf);
            } else {
              tc_commit(empty0 + 8 * s);
              if (kb == kb1 - 1) tc_commit(accfull0 + 8 * buf);
            }
            if (ti == 0 && kb == kb1 - 1) TC_STAMP(p.dbg, 30);
          }
          __syncwarp();
          if (PARTS == 2) { third += 4; while (third >= Cf::NMAIN) third -= Cf::NMAIN; }
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {  // ---------------- epilogue (warps 2-9)
    // Two warps per quarter of the rows take 32-column chunks in turn: TMEM -> registers (thread = accumulator row) -> this warp's
    // staging tile in shared memory (16-byte pieces swizzled by the row: neither way conflicts) -> half warps own rows, lanes
    // adjacent column pairs, so every global access of the fused epilogue is coalesced.
    const int quarter = warp & 3;  // a warp may only touch TMEM lanes 32 * (warp % 4) ..
    const int cfirst = (warp - 2) / 4 * 32;
    float* Cs = reinterpret_cast<float*>(p.smem_raw + (p.epi0 - p.raw)) + (warp - 2) * 32 * 32;
    const int hl = lane & 15, rsub = lane >> 4;  // column pair and row parity of this lane
    auto staged = [&](int i) {                   // its pair in row 2 i + rsub
      const int r = 2 * i + rsub;
      return *reinterpret_cast<const float2*>(Cs + r * 32 + (((hl >> 1) ^ (r & 7)) << 2) + (hl & 1) * 2);
    };
    const int start_pos = (EPI == EPI_ROPE_KV) ? *e.pos_ptr : 0;
    // hands an accumulator buffer back to the products (of a pair: to its first CTA, which waits for both)
    auto hand_back = [&](uint32_t buf) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (CG == 2) pair_arrive(cluster_at(accempty0 + 8 * buf, 0));
        else mbar_arrive(accempty0 + 8 * buf);
      }
    };
    uint32_t ti = 0;
    for (int t = first_tile; t < ntiles; t += tile_stride, ++ti) {
      const int tmn = t % ntiles_mn, ks = t / ntiles_mn, out_tile = tmn * CG + rank;
      const int m0 = (tmn % tiles_m) * TM + rank * Cf::BM, n0 = (tmn / tiles_m) * bn;
      const uint32_t buf = ti % NBUF, use = ti / NBUF;
      mbar_wait(accfull0 + 8 * buf, use & 1, fail);
      tc_fence_after();
      if (ti == 0 && threadIdx.x == 64) TC_STAMP(p.dbg, 32);
      const uint32_t acc = p.tmem_base + buf * ACC_COLS + ((uint32_t)(quarter * 32) << 16);
      const int mq = m0 + quarter * 32, cols = min(bn, N - n0);
      const bool live = mq < rows && cfirst < cols;  // warp-uniform: this warp has something to do
      // accumulator columns c .. c+31 of this thread's row (3xTF32: the accumulators summed)
      auto load_acc = [&](int c, float (&v)[32]) {
        tmem_ld32(acc + (uint32_t)c, v);
        if (Cf::NACC > 1) {  // the main accumulators plus the correction accumulator
#pragma unroll
          for (int k2 = 1; k2 < Cf::NACC; ++k2) {
            float w[32];
            tmem_ld32(acc + (uint32_t)c + k2 * bn, w);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] += w[j];
          }
        }
      };
      // K-split scratch: [k slice][output tile][column / 4][row of the tile] float4, so that a warp's 32 rows are contiguous both ways
      const size_t slice = (size_t)ntiles_mn * CG * (bn / 4) * Cf::BM;
      float4* pt = reinterpret_cast<float4*>(part) + (size_t)out_tile * (bn / 4) * Cf::BM + quarter * 32 + lane;
      if (ksplit > 1) {
        // K-split: publish this slice's partial tile, then the LAST slice to arrive (per output tile)
        // sums all slices in slice order - a fixed order, so the result does not depend on timing -
        // and runs the fused epilogue on the sum.
#pragma unroll 1
        for (int c = cfirst; c < cols; c += 64) {
          if (mq >= rows) break;
          float v[32];
          load_acc(c, v);
#pragma unroll
          for (int j = 0; j < 32; j += 4) __stcg(pt + ks * slice + (size_t)((c + j) / 4) * Cf::BM, make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
        }
        hand_back(buf);
        // As in gemm_swap.cu: the CTA barrier orders the warps' partial stores before thread 64's acq_rel atomic
        // (cumulative release), whose acquire side + the next barrier order the last arriver's reads - instead of two
        // __threadfence() per thread.
        asm volatile("bar.sync 2, 256;" ::: "memory");  // the eight epilogue warps
        int* flag = reinterpret_cast<int*>(p.smem_raw + (p.tmem_slot - p.raw)) + 1;
        if (threadIdx.x == 64) {
          int old;
          asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(tile_cnt + out_tile) : "memory");
          *flag = (old == ksplit - 1);
          if (old == ksplit - 1) tile_cnt[out_tile] = 0;  // ready for the next launch
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
        const bool is_last = *flag != 0;
        asm volatile("bar.sync 2, 256;" ::: "memory");  // everyone has read the flag before it is reused
        if (!is_last) continue;
      }
      if constexpr (EPI == EPI_ARGMAX) {
        if (ksplit == 1) {
          // Greedy argmax fused into the LM head (llama3.py:320) without leaving the registers: a thread IS an
          // accumulator row, so it walks its chunks' columns in increasing order keeping (max, first index) and
          // merges into best[m] with ONE 64-bit atomicMax per tile.  (The shared-memory pass + per-row shuffle
          // tree this replaces took as long as the tile's 108-MMA main loop.)
          float bv = -INFINITY;
          int bi = 0x7fffffff;
#pragma unroll 1
          for (int c = cfirst; c < cols; c += 64) {
            if (mq >= rows) break;  // warp-uniform
            float v[32];
            load_acc(c, v);
            const int cbase = n0 + c;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (cbase + j < N && v[j] > bv) { bv = v[j]; bi = cbase + j; }
          }
          hand_back(buf);
          const int m = mq + lane;
          if (m < rows && bi != 0x7fffffff) atomicMax(e.best + m, argmax_key(bv, e.col_offset + bi));
          continue;
        }
      }
      int row_b = 0, row_pos = -1, row_real = 1;  // lane i: (sequence, position, not padding) of accumulator row quarter * 32 + i
      if (EPI == EPI_ROPE_KV && mq + lane < rows) {
        const int m = mq + lane;
        row_b = m / e.L;
        const int t = m - row_b * e.L;
        row_pos = (e.row_pos ? e.row_pos[row_b] : start_pos) + t;
        row_real = !e.row_len || t < e.row_len[row_b];
      }
#pragma unroll 1
      for (int c0 = cfirst; c0 < cols; c0 += 64) {
        if (!live) break;
        __syncwarp();  // the previous chunk's reads of Cs are done
        {
          float v[32];
          if (ksplit == 1) {
            load_acc(c0, v);
          } else {  // sum of the slices' partials, slice 0 first
            const float4* src = pt + (size_t)(c0 / 4) * Cf::BM;
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.f;
            // three slices' values are requested before the first is added (slice order: the sum does not depend on timing): one L2
            // round trip per three slices.  With one slice ahead of the additions, and rows a tile's width apart, the reading took
            // longer than the main loop it saved
            for (int k2 = 0; k2 < ksplit; k2 += 3) {
              float4 q[3][8];
#pragma unroll
              for (int u = 0; u < 3; ++u)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                  q[u][j] = k2 + u < ksplit ? __ldcg(src + (size_t)(k2 + u) * slice + (size_t)j * Cf::BM) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int u = 0; u < 3; ++u)
#pragma unroll
                for (int j = 0; j < 8; ++j) { v[4 * j] += q[u][j].x; v[4 * j + 1] += q[u][j].y; v[4 * j + 2] += q[u][j].z; v[4 * j + 3] += q[u][j].w; }
            }
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(Cs + lane * 32 + ((j ^ (lane & 7)) << 2)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        if (ksplit == 1 && c0 + 64 >= cols) hand_back(buf);  // last TMEM read of this tile: early
        __syncwarp();
        const int col = n0 + c0 + hl * 2;  // this lane's column pair
        const bool col_ok = col < N, has1 = col + 1 < N;
        const int mr = mq + rsub;          // row of pair i: mr + 2 i
        if constexpr (EPI == EPI_RESID) {
          // x += tile: all rows of this lane are loaded before the first store (one latency)
          if (col_ok) {
            float2 rr[16];
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (mr + 2 * i < rows) rr[i] = *reinterpret_cast<const float2*>(e.resid + (size_t)(mr + 2 * i) * e.ld_out + col);
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (mr + 2 * i < rows) {
                const float2 tt = staged(i);
                *reinterpret_cast<float2*>(e.out + (size_t)(mr + 2 * i) * e.ld_out + col) = make_float2(rr[i].x + tt.x, rr[i].y + tt.y);
              }
          }
        } else if constexpr (EPI == EPI_ARGMAX) {
          // greedy argmax fused into the LM head (llama3.py:320): per row, the chunk's best
          // (value, first index) is merged into best[m] with one 64-bit atomicMax.
#pragma unroll 1
          for (int i = 0; i < 16; ++i) {
            const int m = mr + 2 * i;
            if (mq + 2 * i >= rows) break;
            float bv = -INFINITY;
            int bi = 0x7fffffff;
            if (col_ok) {
              const float2 tt = staged(i);
              bv = tt.x; bi = col;
              if (has1 && tt.y > bv) { bv = tt.y; bi = col + 1; }
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
              const float ov = __shfl_xor_sync(L3_FULL, bv, o);
              const int oi = __shfl_xor_sync(L3_FULL, bi, o);
              if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
            }
            if (hl == 0 && m < rows && bi != 0x7fffffff) atomicMax(e.best + m, argmax_key(bv, e.col_offset + bi));
          }
        } else if constexpr (EPI == EPI_ROPE_KV) {
          // rotate q / k pairs (llama3.py:41-76) and append k, v to the cache (llama3.py:184-185).
          // (sequence, position) of the warp's 32 rows were computed once per tile (row_b, row_pos);
          // what depends on the column alone is computed once per chunk.
          const int qcols = e.HN * e.HD, kcols = e.KVHN * e.HD;
          const int region = col < qcols ? 0 : (col < qcols + kcols ? 1 : 2);
          const int within = region == 0 ? col : (region == 1 ? col - qcols : col - qcols - kcols);
          const int h = within / e.HD, d = within % e.HD, jj = d >> 1, hd2 = e.HD >> 1;
          KVT* cbase = (KVT*)(region == 1 ? e.cache_k : e.cache_v) + (size_t)h * e.M * e.HD + d;
          // The table entries of all rows are requested before the first store: one L2 round trip per chunk
          // instead of one per group of four rows (a load may not move above a store that could alias it) - eight
          // dependent round trips per chunk made this epilogue (11 us per 128 x 256 tile) longer than a K = 2048
          // mainloop.
          float c[16], sn[16];
          const bool rot = region < 2 && col_ok;  // differs between lanes where a chunk straddles the q | k | v borders
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int pi = __shfl_sync(L3_FULL, row_pos, 2 * i + rsub);  // every lane takes part
            const size_t ti = (size_t)max(pi, 0) * hd2 + jj;   // rows beyond the batch: entry of position 0, unused
            c[i] = rot ? __ldg(e.cos_tab + ti) : 1.f;
            sn[i] = rot ? __ldg(e.sin_tab + ti) : 0.f;
          }
#pragma unroll
          for (int rb = 0; rb < 16; rb += 4) {
            if (mq + 2 * rb >= rows) break;
            float2 v[4];
            int pos[4], bb[4], real[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              pos[i] = __shfl_sync(L3_FULL, row_pos, 2 * (rb + i) + rsub);
              bb[i] = __shfl_sync(L3_FULL, row_b, 2 * (rb + i) + rsub);
              real[i] = __shfl_sync(L3_FULL, row_real, 2 * (rb + i) + rsub);
            }
            if (!col_ok) continue;
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = staged(rb + i);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (pos[i] < 0) continue;  // row beyond the batch
              float r0 = v[i].x, r1 = v[i].y;
              if (region < 2) {
                r0 = v[i].x * c[rb + i] - v[i].y * sn[rb + i];
                r1 = v[i].x * sn[rb + i] + v[i].y * c[rb + i];
              }
              if (region == 0) {
                const size_t o = (size_t)(mr + 2 * (rb + i)) * e.ld_out + col;
                if (e.out) *reinterpret_cast<float2*>(e.out + o) = make_float2(r0, r1);
                if (e.out_bf16) *reinterpret_cast<__nv_bfloat162*>(e.out_bf16 + o) = __floats2bfloat162_rn(r0, r1);
              } else if (real[i]) {  // padding tokens of a ragged prefill leave the cache untouched
                KVT* ck = cbase + ((size_t)bb[i] * e.KVHN * e.M + pos[i]) * e.HD;
                if constexpr (sizeof(KVT) == 2) *reinterpret_cast<__nv_bfloat162*>(ck) = __floats2bfloat162_rn(r0, r1);
                else *reinterpret_cast<float2*>(ck) = make_float2(r0, r1);
              }
            }
          }
        } else if constexpr (EPI == EPI_SWIGLU) {
          // h = silu(gate) * up over interleaved (gate_j, up_j) columns (llama3.py:99-101).  bf16 mode
          // uses the fast exponential / reciprocal (its bar is 3e-2) unless glu_exact asks for the full ones; fp32 mode keeps the exact form.
          // All values before the first store, and the activation decided once per chunk: with a store between them the 16
          // exponentials and divisions follow one another (128 x 256 at K = 2048: the epilogue took longer than the products).
          if (col_ok) {
            float hv[16];
            if (e.act == GLU_SILU && !e.glu_w) {
              if (KIND == TC_BF16 && !e.glu_exact) {
#pragma unroll
                for (int i = 0; i < 16; ++i) { const float2 t = staged(i); hv[i] = t.x * __fdividef(1.0f, 1.0f + __expf(-t.x)) * t.y; }
              } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) { const float2 t = staged(i); hv[i] = silu_ref(t.x) * t.y; }
              }
            } else if (!e.glu_w && e.act == GLU_GELU_TANH) {
#pragma unroll
              for (int i = 0; i < 16; ++i) { const float2 t = staged(i); hv[i] = gelu_tanh_ref(t.x) * t.y; }
            } else if (!e.glu_w && e.act == GLU_CLAMP) {
              const float limit = e.act_limit, slope = e.act_slope;
#pragma unroll
              for (int i = 0; i < 16; ++i) { const float2 t = staged(i); hv[i] = glu_clamp<KIND == TC_BF16>(limit, slope, t.x, t.y); }
            } else {
              const int g = e.glu_w ? (col >> 1) / e.glu_group : 0;
              const bool weighted = e.glu_w && g < e.glu_groups;
              float wt[16];
#pragma unroll
              for (int i = 0; i < 16; ++i) wt[i] = weighted && mr + 2 * i < rows ? e.glu_w[(size_t)(mr + 2 * i) * e.glu_w_ld + g] : 1.f;
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                float2 t = staged(i);
                const float wi = e.glu_w_out ? 1.f : wt[i];
                t.x *= wi; t.y *= wi;
                hv[i] = e.act == GLU_SILU && KIND == TC_BF16 && !e.glu_exact ? t.x * __fdividef(1.0f, 1.0f + __expf(-t.x)) * t.y : glu_pair<KIND == TC_BF16>(e, t.x, t.y);
                if (e.glu_w_out) hv[i] *= wt[i];
              }
            }
            const size_t o = (size_t)mr * e.ld_out + (col >> 1);
            if (e.out_lo) {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (mr + 2 * i < rows) split_tf32(hv[i], e.out[o + (size_t)(2 * i) * e.ld_out], e.out_lo[o + (size_t)(2 * i) * e.ld_out]);
            } else if (e.out) {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (mr + 2 * i < rows) e.out[o + (size_t)(2 * i) * e.ld_out] = hv[i];
            }
            if (e.out_bf16) {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (mr + 2 * i < rows) e.out_bf16[o + (size_t)(2 * i) * e.ld_out] = __float2bfloat16_rn(hv[i]);
            }
          }
        } else if (!e.out_lo && !(e.ld_out & 1) && !(N & 1)) {
          // EPI_STORE, whole column pairs: all rows are read from Cs before the first of their stores, row
          // pointers advance by the leading dimension, and what does not depend on the row is decided once per chunk
          const int left = rows - mr;
          if (col_ok) {
            float* po = e.out ? e.out + (size_t)mr * e.ld_out + col : nullptr;
            bf16* pb = e.out_bf16 ? e.out_bf16 + (size_t)mr * e.ld_out + col : nullptr;
            float2 tt[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) tt[i] = staged(i);
            if (e.unary) {
#pragma unroll
              for (int i = 0; i < 16; ++i) { tt[i].x = unary_act(e.unary, tt[i].x); tt[i].y = unary_act(e.unary, tt[i].y); }
            }
            if (po) {
#pragma unroll
              for (int i = 0; i < 16; ++i, po += 2 * e.ld_out)
                if (2 * i < left) *reinterpret_cast<float2*>(po) = tt[i];
            }
            if (pb) {
#pragma unroll
              for (int i = 0; i < 16; ++i, pb += 2 * e.ld_out)
                if (2 * i < left) *reinterpret_cast<__nv_bfloat162*>(pb) = __floats2bfloat162_rn(tt[i].x, tt[i].y);
            }
          }
        } else {  // EPI_STORE, any strides
#pragma unroll 1
          for (int i = 0; i < 16; ++i) {
            const int m = mr + 2 * i;
            if (m >= rows || !col_ok) break;
            const float2 t = staged(i);
            epilogue_pair<KVT>(EPI, e, m, col, t.x, t.y, has1);
          }
        }
      }
      if (ksplit == 1 && !live) hand_back(buf);  // nothing was read
      if (ti == 0 && threadIdx.x == 64) TC_STAMP(p.dbg, 34);
    }
  }
}
