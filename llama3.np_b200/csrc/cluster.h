// Interface of the one-cluster decode step of small fp32 models (decode_cluster.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "mega.h"

struct ClusterArgs {
  const MegaLayer* layers;           // device array [NL], fp32 weights and caches
  int NL, D, HN, KVHN, HD, FD, M, B, vocab;
  const float* embed;
  float eps;
  const float *cos_tab, *sin_tab;
  // token and position of every sequence: ids (non-null) at [b * ids_ld + ids_off], position scal[0]; or the generate loop's next
  // tokens d_next[b] at position scal[2] + scal[1] + 1
  const int32_t* ids;
  int ids_ld, ids_off;
  const int32_t* d_next;
  const int* scal;
  float* x;                          // [B, D] the residual stream behind the last layer
  int* err;                          // mapped host memory: set to 1 when a wait inside the kernel ran out
  bool pdl;                          // starts in its predecessor's tail: weights are drawn ahead
};
struct ClusterHeadArgs {             // next = argmax(norm(x) W^T), then the step's bookkeeping
  const float *x, *w, *norm;
  float eps;
  int B, D, VS, M;
  unsigned long long* best;          // [B] zero between steps
  int* done;                         // [1] zero between steps
  int32_t* d_next;
  int64_t* d_tokens;                 // [B, M]
  int* scal;
  float* logits;                     // [B, VS]: the logits in place of argmax and bookkeeping (null: these)
  int* err;                          // as ClusterArgs::err
};
// most sequences a step can take, 0: the shape or the device is not one for it
int decode_cluster_max_batch(int NL, int D, int HN, int KVHN, int HD, int FD, int M);
cudaError_t launch_decode_cluster(const ClusterArgs& a, cudaStream_t s);
cudaError_t launch_cluster_head(const ClusterHeadArgs& a, int n_sm, cudaStream_t s);
