// Interface of the tcgen05 tensor-core GEMM (gemm_tc.cu).
#pragma once
#include <cuda.h>

#include "common.cuh"

// TC_TF32X3_2: the 3xTF32 scheme with ONE main accumulator instead of three (short K loops: the per-MMA
// truncation drift stays ~2e-6 up to K = 512), half the TMEM columns -> wider / double-buffered tiles
enum TcKind : int { TC_BF16 = 0, TC_TF32X3 = 1, TC_TF32X3_2 = 2 };

struct TcGemmArgs {
  int kind;             // TcKind
  const void* A[2];     // activations [rows, K]: bf16, or fp32 (hi, lo) pair
  const void* W[2];     // weights [N, K], same element kind
  int rows, N, K;
  int bn, ksplit;       // set by the launcher
  int epi;
  EpiArgs e;
  int ldw;              // row stride of W (0: K)
  // bf16: rows in groups that take their own part of W.  groups (device): [0] the number of 128-row tiles, [1 + i] the group g of tile i;
  // a tile's weight rows start at g * group_n, its K range at g * group_k.  W is [w_rows, w_cols]; `rows` is the room of A and of the
  // outputs, group_rows what the caller expects to be used (the choice of the tile width).
  const int* groups;
  int group_n, group_k, w_rows, w_cols, group_rows;
  // optional caller-owned scratch for the deterministic K-split of gemm_tc.cu (null: never split)
  float* part;       // room for ksplit x (rows padded to 128) x (N padded to the tile) fp32 partial sums
  size_t part_bytes;
  int* tile_cnt;     // zero-initialised arrival counters, one per output tile
  int tile_cnt_len;
  int* err;             // gemm_tc.cu: set to 1 when a wait inside the kernel ran out (null: the launch fails)
  bool no_cluster;      // gemm_swap.cu: slices that would be a cluster are published in the scratch instead, for comparisons
};

cudaError_t launch_gemm_tc(const TcGemmArgs& a, cudaStream_t s);
// how a launch cuts its work: CTAs that share a tile, the tile's width (gemm_swap.cu: height), slices of K, and whether slices are added
// in whatever order they arrive
struct TcPlan { int ctas, width, slices, any_order; bool cluster = false; };  // cluster: the slices of a tile are one (gemm_swap.cu)
TcPlan gemm_tc_plan(const TcGemmArgs& a);    // bf16
TcPlan gemm_swap_plan(const TcGemmArgs& a);
// swapped operand roles for 9..128 activation rows (gemm_swap.cu): same arguments
bool gemm_swap_supported(int rows, int N);
cudaError_t launch_gemm_swap(const TcGemmArgs& a, cudaStream_t s);
cudaError_t launch_split_tf32(const float* src, float* hi, float* lo, int64_t n, cudaStream_t s);
bool tc_gemm_supported(int K);
void tc_forget_maps();
int tc_debug_timeline(int enable, unsigned long long* out64);
// cached 2-D tensor map of a row-major [rows, cols] matrix: box = 128 bytes of columns x box_rows rows,
// 128-byte swizzle (null if the driver entry point is unavailable)
// (ld: row stride in elements, 0 = cols; multiples of 16 bytes)
const CUtensorMap* tc_get_map(const void* ptr, bool is_bf16, int rows, int cols, int box_rows, int ld = 0);

// fp32 projections at fp32 precision on the tensor cores (gemm_f32.cu): fp32 A, W fp32 or bf16; EPI_STORE, EPI_RESID, EPI_SWIGLU
struct GemmF32Args {
  const float* A;       // [rows, K], row stride lda (0: K)
  int lda;
  const void* W;        // [N, K]
  bool w_bf16;
  int rows, N, K, epi;
  EpiArgs e;
  float* part;          // scratch of the K split, as TcGemmArgs (null: never split)
  size_t part_bytes;
  int* tile_cnt;
  int tile_cnt_len;
  int* err;             // set to 1 when a wait inside the kernel ran out
  // both operands cut beforehand (launch_cut_rows): planes of [rows, K] and [N, K] bf16 parts, x_plane values apart; A and W as well
  const void *A_planes, *W_planes;
  int64_t a_plane, w_plane;
};
bool gemm_f32_planes_supported(const void* W_planes, int64_t w_plane, int K);
cudaError_t launch_cut_rows(const float* src, int lda, int rows, int K, void* dst, int64_t plane, cudaStream_t s);
const CUtensorMap* tc_get_planes_map(const void* ptr, int rows, int cols, int box_rows, int64_t plane);  // box: 64 columns, three planes
bool gemm_f32_supported(const GemmF32Args& a);
cudaError_t launch_gemm_f32(const GemmF32Args& a, cudaStream_t s);
