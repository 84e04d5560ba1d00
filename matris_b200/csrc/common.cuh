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

// Two float32 values at a time: one instruction where the scalar forms take two, each half rounded as the scalar form rounds it.  The
// warps of the contraction kernels' prologues and epilogues wait for instruction slots as much as for anything else (k_mlp: 13 k
// a scheduler for a tile of 30 k cycles, a third of them float32 additions and products).
struct f2 { unsigned long long v; };
__device__ __forceinline__ f2 two(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void apart(f2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ f2 operator+(f2 a, f2 b) {
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a.v) : "l"(b.v));
  return a;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b) {
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(a.v) : "l"(b.v));
  return a;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(a.v) : "l"(b.v), "l"(c.v));
  return a;
}
__device__ __forceinline__ f2 less(f2 a, f2 b) { return fma2(b, two(-1.f, -1.f), a); }  // a - b
__device__ __forceinline__ f2 low(const float4& v) { return two(v.x, v.y); }
__device__ __forceinline__ f2 high(const float4& v) { return two(v.z, v.w); }
__device__ __forceinline__ f2 sigmoid_fast_2(f2 x) {
  float e0, e1;
  apart(x * two(-1.442695041f, -1.442695041f), e0, e1);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e0));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(e1));
  apart(two(1.f, 1.f) + two(e0, e1), e0, e1);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(e0));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(e1));
  return two(e0, e1);
}
__device__ __forceinline__ f2 silu_fast_2(f2 x) { return x * sigmoid_fast_2(x); }
__device__ __forceinline__ f2 silu_grad_fast_2(f2 x) {
  const f2 s = sigmoid_fast_2(x), one = two(1.f, 1.f);
  return s * fma2(x, less(one, s), one);
}
// x[0..3] += v, *= SiLU'(v), = v w + x, = SiLU(x)
__device__ __forceinline__ void add4_to(float* x, const float4& v) {
  apart(two(x[0], x[1]) + low(v), x[0], x[1]);
  apart(two(x[2], x[3]) + high(v), x[2], x[3]);
}
__device__ __forceinline__ void silu_grad4_to(float* x, const float4& v) {
  apart(two(x[0], x[1]) * silu_grad_fast_2(low(v)), x[0], x[1]);
  apart(two(x[2], x[3]) * silu_grad_fast_2(high(v)), x[2], x[3]);
}
__device__ __forceinline__ void fma4_to(float* x, const float4& v, const float4& w) {
  apart(fma2(low(w), low(v), two(x[0], x[1])), x[0], x[1]);
  apart(fma2(high(w), high(v), two(x[2], x[3])), x[2], x[3]);
}
template <int N> __device__ __forceinline__ void silu_fast_all(const float* x, float (&y)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) apart(silu_fast_2(two(x[i], x[i + 1])), y[i], y[i + 1]);
}

// What the gradient of a row ahead of a gated MLP's tail consists of (row_math.cuh has the expressions)
struct RowGrad {
  int32_t kind;        // 0: dh_in, 1: attention rows, 2: smoothed rows
  int32_t idx_stride;  // of tgt and src
  const float* dh_in; const int32_t* dh_map; float dh_scale;  // given part (kinds 1 and 2: may be NULL)
  const int32_t *tgt, *src, *emap;
  const float *logits, *h, *agg_t, *agg_s, *stats, *dagg_t, *dagg_s;  // kind 1
  float* dlogits;                                                     // kind 1, optional in the few-row product
  const float *env, *dagg;                                            // kind 2
  const float *z2, *norm_core, *norm_gate;                            // the tail: z2 [rows, 256]
};
// The backward pass of a gated MLP from a row's gradient on, for few rows, as one launch: dz2 = tail'(RowGrad) in registers,
// dz1 = (dz2 W2t) SiLU'(z1), and, with n_out > 0, out[j] = dz1 W1t_j (+ dlogits W3t) (+ res_w res, j = 0).  W1t has 128 rows for
// every output.  `zero`: n_zero floats to be cleared on the way (a multiple of 4).
struct RowBwd {
  int64_t n_rows;
  RowGrad g;
  mb_weight w2t, w1t, w3t;  // w3t.W NULL: no logits' share
  const float* z1; float* dz1;
  int32_t n_out;
  float* out[3];
  const float *res, *res_w;
  float* zero; int64_t n_zero;
};
bool few_row_bwd_fits(int64_t n_rows, int n_out, bool logits);  // whether it takes so many rows
int few_row_bwd(const RowBwd& a, cudaStream_t stream);
// n independent mb_gemm problems of few rows as one launch
bool few_linears_fit(const mb_gemm_desc* const* g, int n);
int few_linears(const mb_gemm_desc* const* g, int n, cudaStream_t stream);
// mb_gemm with an operand row that is the sum of rows i and pair[i], i = idx[r]
bool pair_linear_fits(const mb_gemm_desc* g);
int pair_linear(const mb_gemm_desc* g, const int32_t* pair, cudaStream_t stream);
bool few_ffn_bwd_fits(int64_t n_rows_a, int64_t n_rows_b);
int few_ffn_bwd(const mb_mlp_bwd* const* g, cudaStream_t stream);  // two plain data gradients (dx only, no residual) of few rows
// y[i] = x[i] w[i]^T, [n_rows, 7] x [7, 128], for up to MANY_LINEARS problems as one launch
constexpr int MANY_LINEARS = 40;
struct ManyLinears { const float *x[MANY_LINEARS], *w[MANY_LINEARS]; float* y[MANY_LINEARS]; };
int many_small_linears(int64_t n_rows, int n, const ManyLinears& a, cudaStream_t stream);
// d_rbf[b] += denv[b] w for the envelopes' gradient denv, which stays in registers (mb_seg_smooth_sum_bwd_env, then mb_small_linear_bwd)
int smooth_env_bwd_rbf(int32_t n_bonds, const mb_row_graph& g, const float* env, const float* h, const float* dagg, const float* drow,
                       const float* w, float* d_rbf, cudaStream_t stream);

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace mb
