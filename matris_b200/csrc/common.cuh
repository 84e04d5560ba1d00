// Shared helpers for the matris_b200 CUDA sources (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "matris_b200.h"

namespace mb {

// last CUDA error text, per host thread
void set_cuda_error(cudaError_t e, const char* where);

#define MB_CUDA_CHECK(expr)                                  \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) {                                 \
      mb::set_cuda_error(_e, #expr);                         \
      return MB_ERR_CUDA;                                    \
    }                                                        \
  } while (0)

#define MB_LAUNCH_CHECK(name)                                \
  do {                                                       \
    cudaError_t _e = cudaGetLastError();                     \
    if (_e != cudaSuccess) {                                 \
      mb::set_cuda_error(_e, name);                          \
      return MB_ERR_CUDA;                                    \
    }                                                        \
  } while (0)

// Kernels of an evaluation are launched with programmatic stream serialization: a kernel may be scheduled, and set itself up,
// while its predecessor is still running, and waits in pdl_sync() before it touches anything a predecessor wrote (or read).
// Launch gaps and prologues (tensor-memory allocation, barriers) then overlap; on small systems, where a kernel lasts a few
// microseconds, they are most of the time (4 atoms: 8.6 -> 7.2 ms an evaluation).  Weights and constants are read behind the wait
// like everything else: a caller of the C ABI may have written them in the launch before.  Every kernel so launched must call
// pdl_sync().  The first launch behind an event of another stream does without: what it waits for is more than its predecessor.
inline thread_local bool launch_after_event = false;
// Set while an evaluation queues a launch that is not the first on its stream: the weights have not been written since before the
// launch ahead of it (whose blocks passed their own wait before this one's were scheduled), so they may be read before pdl_sync().
inline thread_local bool weights_settled = false;
template <typename... P, typename... A>
static inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = launch_after_event ? 0 : 1;
  launch_after_event = false;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // errors surface in MB_LAUNCH_CHECK
}
// wait for the preceding kernels' results, then let the next kernel be scheduled
__device__ __forceinline__ void pdl_sync() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
}

static inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

int sm_count(int* n);  // multiprocessors of the current device, asked for once per device; a status code
int gemm_mode();  // the contraction core selected with mb_set_gemm_mode

// exclusive scan of n int32 values into out[0..n] (out[n] = total); tmp holds
// mb_graph_scan_tmp_len(n) ints.  in may alias out.
int scan_exclusive(const int32_t* in, int32_t* out, int64_t n, int32_t* tmp, cudaStream_t s);

// accurate expf on purpose: these feed fp32-tolerance parity checks
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
// d/dx [x * sigmoid(x)] = s * (1 + x * (1 - s))   (matris/model/op/fused_silu_op.py:5-13)
__device__ __forceinline__ float silu_grad_f(float x) {
  const float s = 1.0f / (1.0f + expf(-x));
  return s * (1.0f + x * (1.0f - s));
}

// Fast variants for the GEMM prologue / epilogue, where the transcendental cost is paid per operand element: the hardware's
// exponential and reciprocal (a few ulp each, far inside the fp32-tolerance gates), denormal intermediates flushed.  Without
// the flush each of the two costs three more instructions for arguments that only occur where the result is 0 or x anyway.
__device__ __forceinline__ float sigmoid_fast_f(float x) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.442695041f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  return r;
}
__device__ __forceinline__ float silu_fast_f(float x) { return x * sigmoid_fast_f(x); }
__device__ __forceinline__ float silu_grad_fast_f(float x) {
  const float s = sigmoid_fast_f(x);
  return s * fmaf(x, 1.0f - s, 1.0f);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace mb
