// A row's gradients in the backward pass, held by a warp (lane l: channels 4 l .. 4 l + 3): shared by the row kernels and by the
// few-row products that form their operands themselves, so that both give the same bits.
#pragma once
#include <float.h>
#include "common.cuh"

namespace mb {

constexpr float RMS_EPS = FLT_EPSILON;  // nn.RMSNorm(eps=None) uses the dtype's machine epsilon

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 sub4(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }
__device__ __forceinline__ float4 scl4(float4 a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
__device__ __forceinline__ float4 exp4(float4 a) { return make_float4(expf(a.x), expf(a.y), expf(a.z), expf(a.w)); }

// Adjoint of  h = SiLU(RMSNorm(z_core) w_core) * sigmoid(RMSNorm(z_gate) w_gate)  for one row: z = the row's 256 values, g = dh
__device__ __forceinline__ void gate_bwd_row(const float* __restrict__ z, int c, const float* __restrict__ wc,
                                             const float* __restrict__ wg, float4 g, float4& dz_core, float4& dz_gate) {
  const float4 xc = ld4(z + c), xg = ld4(z + 128 + c);
  const float rc = rsqrtf(warp_sum(dot4(xc, xc)) * (1.f / 128.f) + RMS_EPS);
  const float rg = rsqrtf(warp_sum(dot4(xg, xg)) * (1.f / 128.f) + RMS_EPS);
  const float4 gwc = ld4(wc + c), gwg = ld4(wg + c);
  const float4 nc = scl4(xc, rc), ng = scl4(xg, rg);
  const float4 yc = mul4(nc, gwc), yg = mul4(ng, gwg);
  float dnc[4], dng[4];
  const float ycv[4] = {yc.x, yc.y, yc.z, yc.w}, ygv[4] = {yg.x, yg.y, yg.z, yg.w};
  const float gv[4] = {g.x, g.y, g.z, g.w}, wcv[4] = {gwc.x, gwc.y, gwc.z, gwc.w}, wgv[4] = {gwg.x, gwg.y, gwg.z, gwg.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float s = sigmoid_f(ycv[k]), gate = sigmoid_f(ygv[k]);
    const float core = ycv[k] * s, gg = gv[k] * gate;
    dnc[k] = gg * (s * (1.f + ycv[k] * (1.f - s))) * wcv[k];
    dng[k] = gg * core * (1.f - gate) * wgv[k];
  }
  const float4 dn_c = make_float4(dnc[0], dnc[1], dnc[2], dnc[3]), dn_g = make_float4(dng[0], dng[1], dng[2], dng[3]);
  const float mc = warp_sum(dot4(dn_c, nc)) * (1.f / 128.f), mg = warp_sum(dot4(dn_g, ng)) * (1.f / 128.f);
  dz_core = scl4(sub4(dn_c, scl4(nc, mc)), rc);
  dz_gate = scl4(sub4(dn_g, scl4(ng, mg)), rg);
}

// Gradient of a row of the softmax-weighted aggregation: o = dh, the logits' source and target halves in ds, dt
__device__ __forceinline__ void attn_bwd_row(const RowGrad& a, int64_t row, int c, float4& o, float4& ds, float4& dt) {
  const int64_t nt = a.tgt[row * a.idx_stride], ns = a.src[row * a.idx_stride];
  const int64_t er = a.emap ? a.emap[row] : row;
  const float4 xs = ld4(a.logits + er * 256 + c), xt = ld4(a.logits + er * 256 + 128 + c);
  const float4 at = mul4(exp4(sub4(xt, ld4(a.stats + nt * 512 + c))), ld4(a.stats + nt * 512 + 128 + c));
  const float4 as = mul4(exp4(sub4(xs, ld4(a.stats + ns * 512 + 256 + c))), ld4(a.stats + ns * 512 + 384 + c));
  const float4 hv = ld4(a.h + row * 128 + c);
  const float4 gt = mul4(at, ld4(a.dagg_t + nt * 128 + c)), gs = mul4(as, ld4(a.dagg_s + ns * 128 + c));
  o = add4(gt, gs);
  if (a.dh_in) {
    const int64_t mr = a.dh_map ? a.dh_map[row] : row;
    o = add4(o, scl4(ld4(a.dh_in + mr * 128 + c), a.dh_scale));
  }
  ds = mul4(gs, sub4(hv, ld4(a.agg_s + ns * 128 + c)));
  dt = mul4(gt, sub4(hv, ld4(a.agg_t + nt * 128 + c)));
}

// Gradient of a row of the smoothed sum, on top of dh_in where given
__device__ __forceinline__ float4 smooth_bwd_row(const RowGrad& a, int64_t row, int c) {
  const int64_t nt = a.tgt[row * a.idx_stride];
  float4 s;
  if (a.src) s = mul4(ld4(a.env + (int64_t)a.src[row * a.idx_stride] * 128 + c), ld4(a.env + nt * 128 + c));
  else s = ld4(a.env + (int64_t)a.emap[row] * 128 + c);
  float4 o = mul4(ld4(a.dagg + nt * 128 + c), s);
  if (a.dh_in) o = add4(o, ld4(a.dh_in + row * 128 + c));
  return o;
}

}  // namespace mb
