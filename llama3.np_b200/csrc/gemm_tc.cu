// Tensor-core projections for many activation rows: C[M, N] = A[M, K] * W[N, K]^T on the
// 5th-generation tensor cores - tcgen05.mma issued by one thread, operands staged in shared
// memory by TMA (128-byte swizzle), the fp32 accumulator tile in TMEM, read back with
// tcgen05.ld for the fused epilogue (store / residual / SwiGLU / RoPE + KV append).
//
// Two operand kinds:
//   TC_BF16   - bf16 A and W (bf16 mode): one kind::f16 MMA per 16-wide K slice.
//   TC_TF32X3 - fp32 mode.  A plain TF32 MMA keeps 10 mantissa bits and would break the 1e-4
//               logit bar (measured 2e-3), so every fp32 operand is stored as an exact pair
//               hi = x with the low 13 mantissa bits cleared, lo = x - hi, and each K slice
//               issues three kind::tf32 MMAs into the same accumulator:
//               A_lo*W_hi + A_hi*W_lo + A_hi*W_hi.  The dropped A_lo*W_lo term is ~2^-22
//               relative.  The tensor core rounds the accumulator toward zero once per MMA
//               instruction (measured: a single accumulator drifts by ~0.5 ulp per instruction,
//               7e-6 at K = 768), so the K slices are dealt round-robin to THREE main TMEM
//               accumulators and the two correction products go to a fourth; the epilogue adds
//               the four in fp32.  End-to-end logits stay within ~1e-6 of the float64 reference.
//
// Warp roles in a 320-thread CTA:
//   warp 0: TMA producer   warp 1: TMEM allocator + MMA issuer   warps 2-9: epilogue
// synchronised by a STAGES-deep ring of full/empty mbarriers and one accumulator barrier.
#include <cuda.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"
#include "gemm_tc.h"

__device__ unsigned long long g_tc_dbg[64];
static std::atomic<unsigned long long*> g_tc_dbg_to[16];  // where a device's launches leave their timeline, in its own memory (null: nowhere)

#include "gemm_tc_dev.cuh"

// Persistent kernel: every CTA walks output tiles t = blockIdx.x, blockIdx.x + gridDim.x, ... (row
// tile fastest, so the CTAs running at one time share a few weight tiles through L2).  The TMA
// producer and the MMA issuer run ahead across tile boundaries; with two TMEM accumulator buffers
// the epilogue warps drain tile i while the tensor core already works on tile i + 1.
template <int KIND, int BN, int CG, int EPI>
__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1,
               const __grid_constant__ CUtensorMap tmB0, const __grid_constant__ CUtensorMap tmB1,
               int rows, int N, int K, int bn, int a_box_rows, int nst, int ksplit, float* part, int* tile_cnt, int* err,
               unsigned long long* dbg, TcGroups grp, EpiArgs e) {
  extern __shared__ uint8_t smem_raw[];
  pdl_launch();  // the next kernel may start its own prologue now
  if (threadIdx.x == 0) {
    TC_STAMP(dbg, 0);
    // descriptor fetches overlap the barrier set-up (the first TMA otherwise waits ~0.7 us for them)
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA0));
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB0));
    if (KIND != TC_BF16) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmA1));
      asm volatile("prefetch.tensormap [%0];" ::"l"(&tmB1));
    }
  }
  TcPipe p;
  p.dbg = dbg;
  tc_pipe_setup<KIND, BN, CG>(p, smem_raw, nst, BN ? BN : bn);
  tc_pipe_ready(p);
  pdl_wait();  // everything above overlapped the previous kernel; its outputs are visible from here
  if (threadIdx.x == 0) TC_STAMP(dbg, 1);
  tc_gemm_run<KIND, BN, CG, EPI>(p, &tmA0, &tmA1, &tmB0, &tmB1, rows, N, K, a_box_rows, ksplit, part, tile_cnt, grp, e, blockIdx.x / CG, gridDim.x / CG);
  if (threadIdx.x == 64) TC_STAMP(dbg, 34);
  tc_pipe_teardown<KIND, BN, CG>(p, err);
  if (threadIdx.x == 0) TC_STAMP(dbg, 35);
}

// ------------------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  });
  return fn;
}

// [rows, K] row-major matrix, box = 128 bytes of K x box_rows rows, 128-byte swizzle, zero OOB fill
static bool make_map(CUtensorMap* tm, const void* ptr, bool is_bf16, int rows, int K, int box_rows, int ld) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const size_t es = is_bf16 ? 2 : 4;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * es};
  cuuint32_t box[2] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(tm, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                  const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// three planes of a row-major [rows, K] bf16 matrix, box = 64 values of K x box_rows rows x 3
static bool make_planes_map(CUtensorMap* tm, const void* ptr, int rows, int K, int box_rows, int64_t plane) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 3};
  cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)plane * 2};
  cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 3};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct MapCache {
  std::map<std::tuple<const void*, int, int, int, int, int>, CUtensorMap> m;
  std::map<std::tuple<const void*, int, int, int, int64_t>, CUtensorMap> planes;
  const CUtensorMap* get_planes(const void* ptr, int rows, int K, int box_rows, int64_t plane) {
    std::lock_guard<std::mutex> g(mu);
    auto key = std::make_tuple(ptr, rows, K, box_rows, plane);
    auto it = planes.find(key);
    if (it != planes.end()) return &it->second;
    CUtensorMap tm;
    if (!make_planes_map(&tm, ptr, rows, K, box_rows, plane)) return nullptr;
    return &planes.emplace(key, tm).first->second;
  }
  std::mutex mu;
  const CUtensorMap* get(const void* ptr, bool is_bf16, int rows, int K, int box_rows, int ld = 0) {
    std::lock_guard<std::mutex> g(mu);
    if (!ld) ld = K;
    auto key = std::make_tuple(ptr, (int)is_bf16, rows, K, box_rows, ld);
    auto it = m.find(key);
    if (it != m.end()) return &it->second;
    CUtensorMap tm;
    if (!make_map(&tm, ptr, is_bf16, rows, K, box_rows, ld)) return nullptr;
    return &m.emplace(key, tm).first->second;
  }
};
static MapCache g_maps;

const CUtensorMap* tc_get_map(const void* ptr, bool is_bf16, int rows, int cols, int box_rows, int ld) {
  return g_maps.get(ptr, is_bf16, rows, cols, box_rows, ld);
}

const CUtensorMap* tc_get_planes_map(const void* ptr, int rows, int cols, int box_rows, int64_t plane) { return g_maps.get_planes(ptr, rows, cols, box_rows, plane); }

int tc_debug_timeline(int enable, unsigned long long* out64) {
  if (out64 && cudaMemcpyFromSymbol(out64, g_tc_dbg, sizeof(unsigned long long) * 64) != cudaSuccess) return -1;
  unsigned long long z[64] = {0};
  void* p = nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  if (cudaMemcpyToSymbol(g_tc_dbg, z, sizeof z) != cudaSuccess || cudaGetSymbolAddress(&p, g_tc_dbg) != cudaSuccess) return -1;
  g_tc_dbg_to[dev & 15] = enable ? (unsigned long long*)p : nullptr;
  return 0;
}

void tc_forget_maps() {
  std::lock_guard<std::mutex> g(g_maps.mu);
  g_maps.m.clear();
  g_maps.planes.clear();
}

bool tc_gemm_supported(int K) { return K % 8 == 0 && encode_fn() != nullptr; }

static int pick_tf32(int kind, int rows, int N) {
  const int tm = (rows + 127) / 128;
  // 3xTF32 keeps four accumulators per tile: BN = 128 fills the TMEM with ONE buffer (no overlap of
  // epilogue and mainloop), BN = 64 leaves room for two - preferred unless L3_TF32_BN128 is set
  static const bool tf32_128 = getenv("L3_TF32_BN128") && atoi(getenv("L3_TF32_BN128")) != 0;
  if (kind == TC_TF32X3_2) {
    static const int lm_bn = getenv("L3_LM_BN") ? atoi(getenv("L3_LM_BN")) : 256;
    return lm_bn;
  }
  for (int bn = tf32_128 ? 128 : 64; bn > 32; bn >>= 1)
    if ((long)tm * ((N + bn - 1) / bn) >= 120) return bn;
  return 32;
}

static int sm_count() {
  static int n[16] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!n[dev & 15]) cudaDeviceGetAttribute(&n[dev & 15], cudaDevAttrMultiProcessorCount, dev);
  return n[dev & 15] > 0 ? n[dev & 15] : 148;
}

// bf16: CTAs per tile (1, or a pair on 256 rows), tile width and K split together, by the cycles of the busiest CTA.  A k-block (64 of
// K) costs a CTA four MMAs of bn / 2 cycles (mma_probe.cu: 128 at 256 columns, 64 at 128, not below 40 - 48) or its shared memory's
// bandwidth, which the arriving tiles and the products' reads share: measured 583 cycles at 256 columns and 354 at 128 for a CTA alone,
// 500, 390 and 275 at 256, 192 and 128 in a pair, whose CTAs hold half of the weight tile each.  The last tile's epilogue is not
// overlapped, a split adds the partial tiles' way through L2, a pair its barrier at the start.  Any width in steps of 32 is taken, so
// that the tiles of a shape fill the machine's last round.  Over 40 shapes of 130 - 4096 rows (profiles/gemm_cuts.jsonl) the choice is
// 0.8 % behind the best of all cuts in the mean, at most 5 % but for 4096 x 1024 x 1024 (16.5 : 14.5 us); what it gave against single CTAs and widths of 2^n, us (fp32 results; swiglu: bf16): 1462 x 2048 x 8192 66 -> 45,
// 1462 x 16384 x 2048 swiglu 122 -> 73, 4096 x 28672 x 4096 swiglu 700 -> 593 (1.62 PFLOP/s), 4096 x 6144 x 4096 165 -> 138,
// 2048 x 2048 x 8192 59 -> 51, 200 x 6144 x 4096 27 -> 20, 300 x 1024 x 1024 12.5 -> 8.5.
static void pick_bf16(const TcGemmArgs& a, int sms, int* cg_out, int* bn_out, int* ks_out) {
  const int nkb = (a.K + 63) / 64;
  const double per_col = a.epi == EPI_ROPE_KV ? 26 : a.epi == EPI_RESID ? 24 : a.epi == EPI_SWIGLU ? 14 : 20;
  double best = 0;
  const int rows = a.groups ? a.group_rows : a.rows;
  for (int cg = 1; cg <= (rows > 128 && !a.groups ? 2 : 1); ++cg) {
    const int tm = (rows + 128 * cg - 1) / (128 * cg);
    for (int bn = 256; bn >= 32; bn -= 32) {
      const int tn = (a.N + bn - 1) / bn, tiles = tm * tn;
      const double block = std::max(2.0 * bn, cg == 1 ? 128 + 1.79 * bn : 160 + 0.93 * bn), epi = 1500 + per_col * bn;
      for (int ks = 1; ks <= (a.epi == EPI_ARGMAX || a.groups ? 1 : 8); ++ks) {
        const int per = (nkb + ks - 1) / ks;
        if (ks > 1 && (!a.part || !a.tile_cnt || tiles * cg > a.tile_cnt_len || per < 3 || (ks - 1) * per >= nkb ||
                       (size_t)tiles * cg * 128 * bn * sizeof(float) * ks > a.part_bytes)) continue;
        const int rounds = (tiles * ks + sms / cg - 1) / (sms / cg);
        const double main = per * block;
        const double cost = (cg - 1) * 1230 + (rounds - 1) * std::max(main, epi) + main + epi + (ks > 1 ? 1500 + bn * (28.0 + 11.0 * ks) : 0.0);
        if (best == 0 || cost < best * 0.99) { best = cost; *cg_out = cg; *bn_out = bn; *ks_out = ks; }
      }
    }
  }
}

template <int KIND, int BN, int CG, int EPI>
static cudaError_t launch_tc_t(const TcGemmArgs& a, cudaStream_t s) {
  using Cf = TcCfg<KIND, BN, CG>;
  auto kern = gemm_tc_kernel<KIND, BN, CG, EPI>;
  static bool attr_done[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_done[dev & 15]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cf::SMEM_MAX);
    if (e != cudaSuccess) return e;
    attr_done[dev & 15] = true;
  }
  constexpr bool b16 = KIND == TC_BF16;
  const int bn = BN ? BN : a.bn, TM = 128 * CG;
  const int a_box = a.rows >= 128 ? 128 : ((a.rows + 7) & ~7);
  const CUtensorMap* A0 = g_maps.get(a.A[0], b16, a.rows, a.K, a_box);
  const int w_rows = a.groups ? a.w_rows : a.N, w_cols = a.groups ? a.w_cols : a.K;
  const CUtensorMap* B0 = g_maps.get(a.W[0], b16, w_rows, w_cols, bn / CG, a.ldw ? a.ldw : w_cols);
  const CUtensorMap* A1 = Cf::PARTS == 2 ? g_maps.get(a.A[1], b16, a.rows, a.K, a_box) : A0;
  const CUtensorMap* B1 = Cf::PARTS == 2 ? g_maps.get(a.W[1], b16, a.N, a.K, bn / CG) : B0;
  if (!A0 || !B0 || !A1 || !B1) return cudaErrorInvalidValue;
  const int ntiles = ((a.N + bn - 1) / bn) * ((a.rows + TM - 1) / TM);
  const int sms = sm_count();
  const int nkb_all = (a.K + Cf::BK - 1) / Cf::BK;
  // K-split (deterministic, see the epilogue) when the output tiles cover less than half the machine:
  // short-and-wide decode projections (N = D = 288: 18 tiles) otherwise leave most SMs idle while
  // each CTA walks the whole K loop.  Needs caller-owned scratch (TcGemmArgs::part / tile_cnt).
  int ksplit = std::max(1, a.ksplit);
  if (!a.ksplit && a.part && a.tile_cnt && ntiles * 2 <= sms && ntiles <= a.tile_cnt_len) {
    ksplit = std::min(std::min(8, sms / ntiles), nkb_all / 3);
    const size_t need = (size_t)((a.rows + 127) / 128 * 128) * ((a.N + bn - 1) / bn * bn) * sizeof(float);
    while (ksplit > 1 && need * ksplit > a.part_bytes) --ksplit;
    // every slice must own at least one k-block
    while (ksplit > 1 && (ksplit - 1) * ((nkb_all + ksplit - 1) / ksplit) >= nkb_all) --ksplit;
    if (ksplit < 1) ksplit = 1;
  }
  dim3 grid(std::min(ntiles * ksplit, sms / CG) * CG);
  // ring depth: no deeper than the K loop; L3_GEMM_MAXSTAGES caps it further so that two kernels' CTAs
  // fit one SM (programmatic dependent launch can then overlap a kernel's prologue with its predecessor)
  static const int env_st = getenv("L3_GEMM_MAXSTAGES") ? atoi(getenv("L3_GEMM_MAXSTAGES")) : 8;
  const int nkb = (nkb_all + ksplit - 1) / ksplit;
  const int nst = std::max(2, std::min(std::min(Cf::stages(bn), env_st), nkb));
  return launch_kc(kern, grid, dim3(TC_THREADS), (size_t)Cf::smem(bn, nst), s, CG, *A0, *A1, *B0, *B1, a.rows, a.N, a.K, bn, a_box, nst, ksplit, a.part, a.tile_cnt,
                  a.err, g_tc_dbg_to[dev & 15].load(), TcGroups{a.groups, a.group_n, a.group_k}, a.e);
}

template <int KIND, int BN, int CG>
static cudaError_t launch_tc_e(const TcGemmArgs& a, cudaStream_t s) {
  switch (a.epi) {
    case EPI_STORE: return launch_tc_t<KIND, BN, CG, EPI_STORE>(a, s);
    case EPI_RESID: return launch_tc_t<KIND, BN, CG, EPI_RESID>(a, s);
    case EPI_SWIGLU: return launch_tc_t<KIND, BN, CG, EPI_SWIGLU>(a, s);
    case EPI_ARGMAX: return launch_tc_t<KIND, BN, CG, EPI_ARGMAX>(a, s);
    default: return launch_tc_t<KIND, BN, CG, EPI_ROPE_KV>(a, s);
  }
}

TcPlan gemm_tc_plan(const TcGemmArgs& a) {
  TcPlan p{1, 32, 1, 0};
  pick_bf16(a, sm_count(), &p.ctas, &p.width, &p.slices);
  return p;
}

cudaError_t launch_gemm_tc(const TcGemmArgs& args, cudaStream_t s) {
  TcGemmArgs a = args;
  if (a.kind == TC_BF16) {
    const TcPlan p = gemm_tc_plan(a);
    a.bn = p.width; a.ksplit = p.slices;
    return p.ctas == 2 ? launch_tc_e<TC_BF16, 0, 2>(a, s) : launch_tc_e<TC_BF16, 0, 1>(a, s);
  }
  const int bn = pick_tf32(a.kind, a.rows, a.N);
  if (a.kind == TC_TF32X3_2) {  // one main accumulator: only the LM-head epilogues are instantiated
    const bool argmax = a.epi == EPI_ARGMAX;
    switch (bn) {
      case 256: return argmax ? launch_tc_t<TC_TF32X3_2, 256, 1, EPI_ARGMAX>(a, s) : launch_tc_t<TC_TF32X3_2, 256, 1, EPI_STORE>(a, s);
      case 128: return argmax ? launch_tc_t<TC_TF32X3_2, 128, 1, EPI_ARGMAX>(a, s) : launch_tc_t<TC_TF32X3_2, 128, 1, EPI_STORE>(a, s);
      default: return argmax ? launch_tc_t<TC_TF32X3_2, 64, 1, EPI_ARGMAX>(a, s) : launch_tc_t<TC_TF32X3_2, 64, 1, EPI_STORE>(a, s);
    }
  }
  switch (bn) {
    case 128: return launch_tc_e<TC_TF32X3, 128, 1>(a, s);
    case 64: return launch_tc_e<TC_TF32X3, 64, 1>(a, s);
    default: return launch_tc_e<TC_TF32X3, 32, 1>(a, s);
  }
}

// ------------------------------------------------------------------------------ operand preparation
// fp32 -> exact (hi, lo) pair for the 3xTF32 scheme; used for weights at load time.
__global__ void split_tf32_kernel(const float* __restrict__ src, float* __restrict__ hi, float* __restrict__ lo, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float h, l;
    split_tf32(src[i], h, l);
    hi[i] = h;
    lo[i] = l;
  }
}
cudaError_t launch_split_tf32(const float* src, float* hi, float* lo, int64_t n, cudaStream_t s) {
  int grid = (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
  if (grid < 1) grid = 1;
  split_tf32_kernel<<<grid, 256, 0, s>>>(src, hi, lo, n);
  return cudaGetLastError();
}
