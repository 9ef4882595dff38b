// ads_internal.h -- shared host/device helpers of libadseismic_gb300.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>

#include "adseismic_gb300.h"

namespace ads {

// ----- error state (thread-local message, status codes) -------------------
void set_error(const char* fmt, ...);
int fail(int code, const char* fmt, ...);
void note_launches(int64_t n);
// Launches issued while a graph is being captured are counted at replay.
void set_launch_counting(bool on);

// Check a CUDA runtime call; on failure record the message and return
// ADS_ERR_CUDA (or ADS_ERR_NOMEM for allocation failures).
#define ADS_CUDA(call)                                                            \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess) {                                                      \
      return ::ads::fail(e_ == cudaErrorMemoryAllocation ? ADS_ERR_NOMEM          \
                                                         : ADS_ERR_CUDA,          \
                         "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_),  \
                         __FILE__, __LINE__);                                     \
    }                                                                             \
  } while (0)

// Check the launch that was just issued.
#define ADS_LAUNCHED(n)                                                           \
  do {                                                                            \
    cudaError_t e_ = cudaGetLastError();                                          \
    if (e_ != cudaSuccess)                                                        \
      return ::ads::fail(ADS_ERR_CUDA, "kernel launch failed: %s (%s:%d)",        \
                         cudaGetErrorString(e_), __FILE__, __LINE__);             \
    ::ads::note_launches(n);                                                      \
  } while (0)

#define ADS_REQUIRE(cond, ...)                                                    \
  do {                                                                            \
    if (!(cond)) return ::ads::fail(ADS_ERR_INVALID, __VA_ARGS__);                \
  } while (0)

// Fail loudly when no usable device is present (no CPU fallback exists).
int require_device();

// out[e] = (T)(in[e] * scale) for e < n, launched on st (one kernel).
int cast_scaled(float* out, const double* in, int64_t n, double scale, cudaStream_t st);
int cast_scaled(double* out, const double* in, int64_t n, double scale, cudaStream_t st);

// Instantiates and uploads the captured graph g (destroyed either way) for launches on st.
int finish_graph(cudaGraph_t g, cudaStream_t st, cudaGraphExec_t* out);
// What a plan's graphs may hold: a node (a kernel launch of the time loops) takes about
// 4 us of plan creation and, once uploaded, 2.8 KB of device memory, which the plans
// leave free beside their own.  64 shots of 1000 x 500 over 3000 steps: 262,000 nodes,
// 1.0 s and 0.7 GB.  Without a limit 128 shots of up to 1200 x 2000 over up to 6000 steps
// made 2.8 million: 11.8 s, 7.1 GB and 24 GB on the host, for gradients of 8.2 s instead
// of 10.3.
constexpr int64_t kMaxGraphNodes = 400000;
constexpr size_t kGraphNodeBytes = 3072;

inline int64_t div_up(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline int64_t round_up(int64_t a, int64_t b) { return div_up(a, b) * b; }

// Host PML helpers (shared by the C API and the plans).
void acoustic_pml_1d(int64_t NX, int64_t NY, double hx, double hy, int64_t npml,
                     double vp_ref, double Rcoef, int use_pml, double* sx, double* ty);
void elastic_cpml(int64_t NX, int64_t NY, double dx, double dy, double dt, int64_t npml,
                  double npower, double k_max, double alpha_max, double vp_ref,
                  double Rcoef, int use_pml, double* ax, double* bx, double* kx,
                  double* ay, double* by, double* ky);

// ---------------------------------------------------------------------------
// Programmatic dependent launch, for the chains of short kernels that a plan's time
// loop is: launch_chained lets the kernel's blocks start while the previous kernel
// of the stream still runs; grid_wait holds a thread until that kernel is complete
// and its writes are visible, so before it a kernel may read only what the time
// loop never writes (items, shot records, tables) and must write nothing.
// grid_release lets the next kernel's blocks start; after grid_wait, so at most
// one kernel waits ahead.  Every thread calls both.  Inside stream capture the
// launches become programmatic graph edges.
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(a)...);
}
#endif

// ---------------------------------------------------------------------------
// Internal grid layout used by the plans: each padded row of ny+2 cells is
// stored with a pitch that is a multiple of 32 elements and an offset of
// JOFF = 31, so that interior column j = 1 starts on a 32-element boundary
// (128 B for FP32, 256 B for FP64) and every warp row load is aligned.  The
// pitch leaves at least 32 spare elements after column ny+1 so that a
// thread's vector load starting at a valid column never leaves its row.
// ---------------------------------------------------------------------------
constexpr int JOFF = 31;
inline int64_t grid_pitch(int64_t ny) { return round_up(ny + 2 + JOFF + 32, 32); }

}  // namespace ads
