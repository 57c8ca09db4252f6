// Error / launch bookkeeping shared by the files that implement the C-ABI (l3_api.cu, layerlist.cu).
#pragma once
#include <cuda_runtime.h>

#include "model.h"

void set_err(L3Model* m, const char* fmt, ...);  // l3_api.cu
int make_err_word(L3Model* m);                   // L3Model::h_err
int check_waits(L3Model* m);                     // behind a synchronisation: did a kernel of the calls before it give up waiting?
// The calling thread's launches are programmatic dependents of their predecessors for as long as this lives (where it pays; see pdl_pays)
struct PdlScope {
  const bool before;
  PdlScope(const L3Model* m, bool pays);
  ~PdlScope();
};
extern const bool g_l3_debug_sync;               // L3_DEBUG_SYNC=1: synchronise after every launch

#define CK(m, call)                                                                         \
  do {                                                                                      \
    cudaError_t e__ = (call);                                                               \
    if (e__ != cudaSuccess) {                                                               \
      set_err(m, "CUDA error %s at %s:%d: %s", cudaGetErrorName(e__), __FILE__, __LINE__,   \
              cudaGetErrorString(e__));                                                     \
      return L3_ECUDA;                                                                      \
    }                                                                                       \
  } while (0)
// a kernel launch: counted (gpu_launches in bench.py is this counter)
#define LAUNCH(m, call)                                                                        \
  do {                                                                                         \
    CK(m, call);                                                                               \
    (m)->launch_acc += 1;                                                                      \
    if (g_l3_debug_sync) { /* L3_DEBUG_SYNC=1: attribute an asynchronous fault to its launch */ \
      cudaError_t e2__ = cudaStreamSynchronize((m)->stream);                                   \
      if (e2__ != cudaSuccess) {                                                               \
        set_err(m, "kernel launched at %s:%d (launch #%lld) failed: %s", __FILE__, __LINE__,   \
                (long long)(m)->launch_acc, cudaGetErrorString(e2__));                         \
        return L3_ECUDA;                                                                       \
      }                                                                                        \
    }                                                                                          \
  } while (0)
#define REQUIRE(m, cond, ...)    \
  do {                           \
    if (!(cond)) {               \
      set_err(m, __VA_ARGS__);   \
      return L3_EINVAL;          \
    }                            \
  } while (0)
