// Row-wise and segment kernels of the interaction blocks (HBM-bound).
//
// Layout: every feature tensor is float32 row-major with 128 channels.  One warp
// owns one row (or one segment); lane l holds channels 4l..4l+3 as a float4, so a
// row is one coalesced 512-byte access and row reductions are warp shuffles.
// Segment reductions walk CSR ranges (rows are stored grouped by target node;
// the source-side grouping is a permutation), so they need no atomics and their
// summation order is fixed.  The one exception is k_seg_sum's third sum, over
// the rows of a centre atom, which adds finished pieces with atomics.
#include "row_math.cuh"

namespace mb {

constexpr int RW_THREADS = 256;
__device__ __forceinline__ float4 fma4(float4 a, float4 b, float4 c) {
  return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w));
}
__device__ __forceinline__ float4 max4(float4 a, float4 b) {
  return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
}
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

#define MB_ROW_PROLOGUE(n_rows)                                                       \
  const int lane = threadIdx.x & 31;                                                  \
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;          \
  if (row >= (n_rows)) return;                                                        \
  const int c = lane * 4;                                                             \
  (void)c;

static inline unsigned row_grid(int64_t n_rows) { return (unsigned)((n_rows * 32 + RW_THREADS - 1) / RW_THREADS); }

// ------------------------------------------------------------------ gated MLP tail
__global__ void k_gate_fwd(int64_t n_rows, const float* __restrict__ z, const float* __restrict__ wc,
                           const float* __restrict__ wg, float* __restrict__ h, const float* __restrict__ res,
                           const float* __restrict__ res_w, float* __restrict__ out2) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float4 xc = ld4(z + row * 256 + c), xg = ld4(z + row * 256 + 128 + c);
  const float rc = rsqrtf(warp_sum(dot4(xc, xc)) * (1.f / 128.f) + RMS_EPS);
  const float rg = rsqrtf(warp_sum(dot4(xg, xg)) * (1.f / 128.f) + RMS_EPS);
  const float4 yc = mul4(scl4(xc, rc), ld4(wc + c)), yg = mul4(scl4(xg, rg), ld4(wg + c));
  const float4 o = make_float4(silu_f(yc.x) * sigmoid_f(yg.x), silu_f(yc.y) * sigmoid_f(yg.y),
                               silu_f(yc.z) * sigmoid_f(yg.z), silu_f(yc.w) * sigmoid_f(yg.w));
  if (h) st4(h + row * 128 + c, o);
  if (out2) {
    float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
    if (res_w) w = ld4(res_w + c);
    st4(out2 + row * 128 + c, fma4(w, ld4(res + row * 128 + c), o));
  }
}

__global__ void k_gate_bwd(int64_t n_rows, const float* __restrict__ z, const float* __restrict__ wc,
                           const float* __restrict__ wg, const float* __restrict__ dh, float* __restrict__ dz) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  float4 dc, dg;
  gate_bwd_row(z + row * 256, c, wc, wg, ld4(dh + row * 128 + c), dc, dg);
  st4(dz + row * 256 + c, dc);
  st4(dz + row * 256 + 128 + c, dg);
}

// ------------------------------------------------------------------ attention aggregation
// One (node, side) per WARPS warps: side 0 the target segment (contiguous rows), side 1 the source segment (through perm).  A warp
// takes batches of rows whose index and data loads are issued together and keeps a running maximum, so that every row is read
// once whatever the segment's length; WARPS = 4 splits the long segments of an atom graph (30 - 80 edges), which a warp alone would
// walk for tens of microseconds, and joins the partial softmax sums in shared memory.
// Latency of the gathered rows bounds it.  Line graph of 117,048 bonds / 522,844 angles (4.5 rows a segment): 350 us with one warp
// walking a segment in two passes, 295 with batches of eight rows, 233 with four (64 registers, twice the warps).  Atom graph of
// 9372 atoms / 234,096 edges 103 -> 105 us (eight warps: 124), of 32 atoms a third of the time.
template <int WARPS>
__global__ void __launch_bounds__(WARPS == 1 ? RW_THREADS : 128, WARPS == 1 ? 4 : 5)
k_seg_attn_fwd(int n_nodes, const int32_t* __restrict__ tgt_ptr, const int32_t* __restrict__ src_ptr,
               const int32_t* __restrict__ src_perm, const int32_t* __restrict__ emap,
               const float* __restrict__ logits, const float* __restrict__ h,
               float* __restrict__ agg_t, float* __restrict__ agg_s, float* __restrict__ stats) {
  pdl_sync();
  constexpr int NB = WARPS == 1 ? 4 : 8;
  __shared__ float4 part[WARPS > 1 ? 3 : 1][WARPS > 1 ? WARPS : 1][WARPS > 1 ? 32 : 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = lane * 4;
  const int64_t item = WARPS > 1 ? (int64_t)blockIdx.x : ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t row = item >> 1;
  const int side = (int)(item & 1);
  if (row >= n_nodes) return;
  const int32_t* ptr = side == 0 ? tgt_ptr : src_ptr;
  const int q0 = ptr[row], q1 = ptr[row + 1];
  const int lcol = side == 0 ? 128 : 0;
  // (not -inf: a batch whose logits are all -inf would rescale by exp(-inf + inf))
  float4 mx = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX);
  float4 s = zero4(), acc = zero4();
  for (int q = q0 + (WARPS > 1 ? w * NB : 0); q < q1; q += NB * WARPS) {
    int64_t r[NB], er[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {  // rows past the end repeat the last one
      const int qq = q + i < q1 ? q + i : q1 - 1;
      r[i] = side == 0 ? qq : src_perm[qq];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) er[i] = emap ? emap[r[i]] : r[i];
    float4 x[NB], hv[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) x[i] = ld4(logits + er[i] * 256 + lcol + c);
#pragma unroll
    for (int i = 0; i < NB; ++i) hv[i] = ld4(h + r[i] * 128 + c);
    float4 m = mx;
#pragma unroll
    for (int i = 0; i < NB; ++i) m = max4(m, x[i]);
    if (q >= q0 + NB * WARPS) {  // a later batch: what has been summed so far was relative to the old maximum
      const float4 f = exp4(sub4(mx, m));
      s = mul4(s, f);
      acc = mul4(acc, f);
    }
    mx = m;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      if (q + i < q1) {
        const float4 e = exp4(sub4(x[i], mx));
        s = add4(s, e);
        acc = fma4(e, hv[i], acc);
      }
    }
  }
  if (WARPS > 1) {
    part[0][w][lane] = mx;
    part[1][w][lane] = s;
    part[2][w][lane] = acc;
    __syncthreads();
    if (w > 0) return;
    const int used = (q1 - q0 + NB - 1) / NB < WARPS ? (q1 - q0 + NB - 1) / NB : WARPS;  // warps that had rows
    for (int k = 1; k < used; ++k) mx = max4(mx, part[0][k][lane]);
    s = acc = zero4();
    for (int k = 0; k < used; ++k) {
      const float4 f = exp4(sub4(part[0][k][lane], mx));
      s = fma4(f, part[1][k][lane], s);
      acc = fma4(f, part[2][k][lane], acc);
    }
  }
  float4 inv = zero4();
  if (q1 > q0) inv = make_float4(1.f / s.x, 1.f / s.y, 1.f / s.z, 1.f / s.w);
  else mx = zero4();
  st4((side == 0 ? agg_t : agg_s) + row * 128 + c, mul4(acc, inv));
  st4(stats + row * 512 + side * 256 + c, mx);
  st4(stats + row * 512 + side * 256 + 128 + c, inv);
}

// Latency of the gathered rows bounds it (5 TB/s of DRAM traffic at half occupancy): six blocks per SM, even with a few spills, beat
// what 62 registers allow.  522,844 angles 579 -> 526 us, 234,096 edges 252 -> 229; eight blocks 557 and 242.
__global__ void __launch_bounds__(RW_THREADS, 6)
k_seg_attn_bwd(int64_t n_rows, const RowGrad a, float* __restrict__ dh, float* __restrict__ gate_dz) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  float4 o, ds, dt;
  attn_bwd_row(a, row, c, o, ds, dt);
  if (gate_dz) {  // dh goes on in registers
    float4 dc, dg;
    gate_bwd_row(a.z2 + row * 256, c, a.norm_core, a.norm_gate, o, dc, dg);
    st4(gate_dz + row * 256 + c, dc);
    st4(gate_dz + row * 256 + 128 + c, dg);
  } else {
    st4(dh + row * 128 + c, o);
  }
  st4(a.dlogits + row * 256 + c, ds);
  st4(a.dlogits + row * 256 + 128 + c, dt);
}

// ------------------------------------------------------------------ refinement aggregation
// WARPS warps per node as in k_seg_attn_fwd (eight: a row costs less here), four rows of a warp in flight: 124 -> 82 us for the line
// graph of 522,844 angles, 47 us as before for the atom graph of 9372 atoms
template <int WARPS>
__global__ void k_seg_smooth_sum_fwd(int n_nodes, const int32_t* __restrict__ tgt_ptr,
                                     const int32_t* __restrict__ emap, const int32_t* __restrict__ src,
                                     int idx_stride, const float* __restrict__ env, const float* __restrict__ h,
                                     float* __restrict__ agg) {
  pdl_sync();
  constexpr int NB = 4;
  __shared__ float4 part[WARPS > 1 ? WARPS : 1][WARPS > 1 ? 32 : 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = lane * 4;
  const int64_t row = WARPS > 1 ? (int64_t)blockIdx.x : ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= n_nodes) return;
  const int q0 = tgt_ptr[row], q1 = tgt_ptr[row + 1];
  float4 acc = zero4();
  for (int q = q0 + (WARPS > 1 ? w * NB : 0); q < q1; q += NB * WARPS) {
    int64_t er[NB];
    float4 hv[NB], ev[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int64_t r = q + i < q1 ? q + i : q1 - 1;
      er[i] = src ? src[r * idx_stride] : emap[r];
      hv[i] = ld4(h + r * 128 + c);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) ev[i] = ld4(env + er[i] * 128 + c);
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (q + i < q1) acc = fma4(hv[i], ev[i], acc);
  }
  if (WARPS > 1) {
    part[w][lane] = acc;
    __syncthreads();
    if (w > 0) return;
#pragma unroll
    for (int k = 1; k < WARPS; ++k) acc = add4(acc, part[k][lane]);
  }
  if (src && q1 > q0) acc = mul4(acc, ld4(env + row * 128 + c));  // line graph: s = env[src] * env[target]
  st4(agg + row * 128 + c, acc);
}

// Bounded by latency like k_seg_attn_bwd; the exponentials of the gate's adjoint come next.  522,844 angles with the adjoint: one
// sigmoid per branch instead of three in all 351 -> 301 us, eight blocks per SM 274 us; 234,096 edges 156 -> 125.
__global__ void __launch_bounds__(RW_THREADS, 8)
k_seg_smooth_sum_bwd_rows(int64_t n_rows, const RowGrad a, float* __restrict__ dh, float* __restrict__ gate_dz) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float4 o = smooth_bwd_row(a, row, c);
  if (gate_dz) {  // dh goes on in registers
    float4 dc, dg;
    gate_bwd_row(a.z2 + row * 256, c, a.norm_core, a.norm_gate, o, dc, dg);
    st4(gate_dz + row * 256 + c, dc);
    st4(gate_dz + row * 256 + 128 + c, dg);
  } else {
    st4(dh + row * 128 + c, o);
  }
}

__device__ __forceinline__ float4 smooth_env_bwd_atom(int64_t row, int c, const int32_t* __restrict__ u2d, const int32_t* __restrict__ rev,
                                                      const int32_t* __restrict__ tgt, const float* __restrict__ h,
                                                      const float* __restrict__ dagg, const float* __restrict__ drow) {
  const int64_t e1 = u2d[row], e2 = rev[e1];
  float4 g1 = ld4(dagg + (int64_t)tgt[e1] * 128 + c), g2 = ld4(dagg + (int64_t)tgt[e2] * 128 + c);
  if (drow) {  // gradient that reached the smoothed rows directly (edge FFN fed with h * s)
    g1 = add4(g1, ld4(drow + e1 * 128 + c));
    g2 = add4(g2, ld4(drow + e2 * 128 + c));
  }
  return add4(mul4(g1, ld4(h + e1 * 128 + c)), mul4(g2, ld4(h + e2 * 128 + c)));
}
__global__ void k_smooth_env_bwd_atom(int n_bonds, const int32_t* __restrict__ u2d, const int32_t* __restrict__ rev,
                                      const int32_t* __restrict__ tgt, const float* __restrict__ h,
                                      const float* __restrict__ dagg, const float* __restrict__ drow,
                                      float* __restrict__ denv) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_bonds)
  st4(denv + row * 128 + c, smooth_env_bwd_atom(row, c, u2d, rev, tgt, h, dagg, drow));
}
// dx[row, 0:7] += v w for a row v held by a warp (w [128, 7]), products and additions in the order of k_small_linear_bwd
__device__ __forceinline__ void row_times_small(int64_t row, int lane, float4 v, const float* __restrict__ w, float* __restrict__ dx) {
  float wr[28];  // of this lane's four channels
#pragma unroll
  for (int i = 0; i < 7; ++i) *reinterpret_cast<float4*>(wr + 4 * i) = ld4(w + 28 * lane + 4 * i);
  float p[8];
#pragma unroll
  for (int j = 0; j < 7; ++j) p[j] = dot4(v, make_float4(wr[j], wr[7 + j], wr[14 + j], wr[21 + j]));
  p[7] = 0.f;
  int o = 16;
#pragma unroll
  for (int n = 4; n > 0; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float keep = up ? p[i + n] : p[i], give = up ? p[i] : p[i + n];
      p[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  for (; o > 0; o >>= 1) p[0] += __shfl_xor_sync(0xffffffffu, p[0], o);
  const int j = lane >> 2;
  if ((lane & 3) == 0 && j < 7) dx[row * 7 + j] = p[0] + dx[row * 7 + j];
}
// The envelopes' gradient straight on into the radial basis's: for few bonds one launch and no denv instead of two.
__global__ void __launch_bounds__(RW_THREADS) k_smooth_env_bwd_atom_rbf(int n_bonds, const int32_t* __restrict__ u2d, const int32_t* __restrict__ rev,
                                          const int32_t* __restrict__ tgt, const float* __restrict__ h,
                                          const float* __restrict__ dagg, const float* __restrict__ drow,
                                          const float* __restrict__ w, float* __restrict__ d_rbf) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_bonds)
  row_times_small(row, lane, smooth_env_bwd_atom(row, c, u2d, rev, tgt, h, dagg, drow), w, d_rbf);
}

// y[r] = x[r] * s[idx[r]]  (rows scaled channel-wise by a gathered row)
__global__ void k_mul_rows_gather(int64_t n_rows, const float* __restrict__ x, const float* __restrict__ s,
                                  const int32_t* __restrict__ idx, float* __restrict__ y) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const int64_t sr = idx ? idx[row] : row;
  st4(y + row * 128 + c, mul4(ld4(x + row * 128 + c), ld4(s + sr * 128 + c)));
}

// done(sum) is called inside: a value that is returned and then stored costs k_smooth_env_bwd_line, at its 40 registers, 24 bytes of
// spills instead of 8 (119,899 bonds / 573,894 angles: 127 us instead of 116).
template <int NB, typename F>  // NB: rows in flight
__device__ __forceinline__ void smooth_env_bwd_line(F done, int64_t row, int c, const int32_t* __restrict__ tgt_ptr,
                                                    const int32_t* __restrict__ src_ptr, const int32_t* __restrict__ src_perm,
                                                    const int32_t* __restrict__ tgt, const int32_t* __restrict__ src,
                                                    int idx_stride, const float* __restrict__ env, const float* __restrict__ h,
                                                    const float* __restrict__ dagg) {
  float4 acc = zero4();
  const int q0 = tgt_ptr[row], q1 = tgt_ptr[row + 1];
  for (int q = q0; q < q1; q += NB) {
    float4 hv[NB], ev[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int64_t r = q + i < q1 ? q + i : q1 - 1;
      ev[i] = ld4(env + (int64_t)src[r * idx_stride] * 128 + c);
      hv[i] = ld4(h + r * 128 + c);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (q + i < q1) acc = fma4(hv[i], ev[i], acc);
  }
  if (q1 > q0) acc = mul4(ld4(dagg + row * 128 + c), acc);
  const int s0 = src_ptr[row], s1 = src_ptr[row + 1];
  for (int q = s0; q < s1; q += NB) {
    int64_t r[NB], nt[NB];
    float4 gv[NB], hv[NB], ev[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) r[i] = src_perm[q + i < s1 ? q + i : s1 - 1];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      nt[i] = tgt[r[i] * idx_stride];
      hv[i] = ld4(h + r[i] * 128 + c);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      gv[i] = ld4(dagg + nt[i] * 128 + c);
      ev[i] = ld4(env + nt[i] * 128 + c);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (q + i < s1) acc = fma4(mul4(gv[i], hv[i]), ev[i], acc);
  }
  done(acc);
}
// Four rows in flight and six blocks per SM (40 registers): 180 -> 121 us for 117,048 bonds / 522,844 angles (four blocks 156).
__global__ void __launch_bounds__(RW_THREADS, 6)
k_smooth_env_bwd_line(int n_nodes, const int32_t* __restrict__ tgt_ptr,
                      const int32_t* __restrict__ src_ptr, const int32_t* __restrict__ src_perm,
                      const int32_t* __restrict__ tgt, const int32_t* __restrict__ src,
                      int idx_stride, const float* __restrict__ env, const float* __restrict__ h,
                      const float* __restrict__ dagg, float* __restrict__ denv) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_nodes)
  smooth_env_bwd_line<4>([&](float4 sum) { st4(denv + row * 128 + c, sum); }, row, c, tgt_ptr, src_ptr, src_perm, tgt, src, idx_stride,
                         env, h, dagg);
}
// For few bonds (see k_smooth_env_bwd_atom_rbf) a warp's chain counts, not the rows in flight on a multiprocessor: eight of them.
__global__ void __launch_bounds__(RW_THREADS, 2)
k_smooth_env_bwd_line_rbf(int n_nodes, const int32_t* __restrict__ tgt_ptr, const int32_t* __restrict__ src_ptr,
                          const int32_t* __restrict__ src_perm, const int32_t* __restrict__ tgt, const int32_t* __restrict__ src,
                          const float* __restrict__ env, const float* __restrict__ h, const float* __restrict__ dagg,
                          const float* __restrict__ w, float* __restrict__ d_rbf) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_nodes)
  smooth_env_bwd_line<8>([&](float4 sum) { row_times_small(row, lane, sum, w, d_rbf); }, row, c, tgt_ptr, src_ptr, src_perm, tgt, src, 1,
                         env, h, dagg);
}

// ------------------------------------------------------------------ sums of row gradients over a node's rows
// out[n, 0:256] = sum of x over the rows whose target is n (contiguous), out[n, 256:512] = over the rows whose source is n
// (through the permutation); with ctr, ctr_out[ctr[r]] += x[r] on top (the rows of a target bond change their centre atom
// at most once, so that is one or two reductions a segment).  The gradient of a node's layer-1 table is exactly these sums: the
// products with the weights then run once per node instead of scattering 128 finished columns per row.
// WARPS warps share a segment: one for the line graph's short segments, eight for an atom's 30 - 80 edges, whose few
// segments would otherwise be walked by a handful of warps.
// 117,048 bonds 178 -> 162 us with four blocks per SM (five: 193, spilling), 9372 atoms 73 -> 62 with eight.
template <int WARPS>
__global__ void __launch_bounds__(256, WARPS == 1 ? 4 : 8)
k_seg_sum(int n_nodes, const int32_t* __restrict__ tgt_ptr, const int32_t* __restrict__ src_ptr,
          const int32_t* __restrict__ src_perm, const int32_t* __restrict__ ctr,
          const float* __restrict__ x, float* __restrict__ out, float* __restrict__ ctr_out) {
  pdl_sync();
  constexpr int NB = 4;  // rows in flight per warp
  __shared__ float4 part[WARPS > 1 ? WARPS : 1][WARPS > 1 ? 64 : 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t item = WARPS > 1 ? (int64_t)blockIdx.x : ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t node = item >> 1;
  const int side = (int)(item & 1), c = lane * 4;
  if (node >= n_nodes) return;
  const int32_t* ptr = side == 0 ? tgt_ptr : src_ptr;
  const int q0 = ptr[node], q1 = ptr[node + 1];
  float4 a = zero4(), b = zero4(), ca = zero4(), cb = zero4();
  const bool by_ctr = WARPS == 1 && side == 0 && ctr != nullptr;
  int cur = -1;
  auto flush = [&]() {
    if (cur < 0) return;
    atomicAdd(reinterpret_cast<float4*>(ctr_out + (int64_t)cur * 256 + c), ca);
    atomicAdd(reinterpret_cast<float4*>(ctr_out + (int64_t)cur * 256 + 128 + c), cb);
    ca = cb = zero4();
  };
  for (int q = q0 + (WARPS > 1 ? w * NB : 0); q < q1; q += NB * WARPS) {
    int64_t r[NB];
    float4 va[NB], vb[NB];
    int ct[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int qq = q + i < q1 ? q + i : q1 - 1;
      r[i] = side == 0 ? qq : src_perm[qq];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      va[i] = ld4(x + r[i] * 256 + c);
      vb[i] = ld4(x + r[i] * 256 + 128 + c);
      ct[i] = by_ctr ? ctr[r[i]] : 0;
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      if (q + i >= q1) break;
      a = add4(a, va[i]);
      b = add4(b, vb[i]);
      if (by_ctr) {
        if (ct[i] != cur) { flush(); cur = ct[i]; }
        ca = add4(ca, va[i]);
        cb = add4(cb, vb[i]);
      }
    }
  }
  if (by_ctr) flush();
  float* const o = out + node * 512 + side * 256;
  if (WARPS > 1) {
    part[w][lane] = a;
    part[w][32 + lane] = b;
    __syncthreads();
    if (threadIdx.x < 64) {
      float4 s = part[0][threadIdx.x];
#pragma unroll
      for (int k = 1; k < WARPS; ++k) s = add4(s, part[k][threadIdx.x]);
      st4(o + 4 * threadIdx.x, s);
    }
  } else {
    st4(o + c, a);
    st4(o + 128 + c, b);
  }
}

// out[u, 0:256] = a[e1] + a[e2] and, with b, out[u, 256:512] = b[e1] + b[e2]: the two directed rows e1, e2 of bond u
__global__ void k_pair_sum(int n_bonds, const int32_t* __restrict__ u2d, const int32_t* __restrict__ rev,
                           const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, int ld) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_bonds)
  const int64_t e1 = u2d[row], e2 = rev[e1];
#pragma unroll
  for (int h = 0; h < 2; ++h)
    st4(out + row * ld + 128 * h + c, add4(ld4(a + e1 * 256 + 128 * h + c), ld4(a + e2 * 256 + 128 * h + c)));
  if (!b) return;
#pragma unroll
  for (int h = 0; h < 2; ++h)
    st4(out + row * ld + 256 + 128 * h + c, add4(ld4(b + e1 * 256 + 128 * h + c), ld4(b + e2 * 256 + 128 * h + c)));
}

// ------------------------------------------------------------------ pair mean / scaling
__global__ void k_pair_mean_res(int n_bonds, const int32_t* __restrict__ u2d, const int32_t* __restrict__ rev,
                                const float* __restrict__ y, const float* __restrict__ res,
                                const float* __restrict__ res_w, float* __restrict__ out) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_bonds)
  const int64_t e1 = u2d[row], e2 = rev[e1];
  float4 o = scl4(add4(ld4(y + e1 * 128 + c), ld4(y + e2 * 128 + c)), 0.5f);
  if (res) {
    float4 w = make_float4(1.f, 1.f, 1.f, 1.f);
    if (res_w) w = ld4(res_w + c);
    o = fma4(w, ld4(res + row * 128 + c), o);
  }
  st4(out + row * 128 + c, o);
}

__global__ void k_scale_rows(int64_t n_rows, const float* __restrict__ x, const float* __restrict__ a,
                             float* __restrict__ y, int accumulate) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  float4 o = ld4(x + row * 128 + c);
  if (a) o = mul4(ld4(a + c), o);
  if (accumulate) o = add4(o, ld4(y + row * 128 + c));
  st4(y + row * 128 + c, o);
}

// ------------------------------------------------------------------ K <= 16 linear layers
// A lane owns four of the 128 columns with their KP (k padded to 8 or 16) weights in registers, loaded once per warp, and a warp takes
// 32 / KP rows at a time: a row is then KP broadcasts and 4 KP products.  (One row per warp with the weights in shared memory, set
// up by every block of eight rows, cost more than the rows: 69 -> 27 us forward and 71 -> 28 backward, on average over the calls of
// 522,844 angles and 117,048 bonds.)
template <int KP>
__device__ __forceinline__ void small_linear_weights(const float* __restrict__ w, int k, int c, float4 (&wr)[KP]) {
  __shared__ float ws[KP][128];  // transposed, so that a warp reads its weights a row at a time
  for (int i = threadIdx.x; i < 128 * k; i += blockDim.x) ws[i % k][i / k] = w[i];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < KP; ++j) wr[j] = j < k ? ld4(&ws[j][c]) : zero4();
}

template <int KP>
__device__ __forceinline__ void small_linear_fwd(int64_t n_rows, int k, const float* __restrict__ x, const float* __restrict__ w,
                                                 float* __restrict__ y) {
  constexpr int ROWS = 32 / KP;
  const int lane = threadIdx.x & 31, c = lane * 4, ri = lane / KP, rj = lane % KP;
  const int64_t step = ((int64_t)gridDim.x * blockDim.x >> 5) * ROWS;
  float4 wr[KP];
  small_linear_weights<KP>(w, k, c, wr);
  for (int64_t r0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * ROWS; r0 < n_rows; r0 += step) {
    const float xv = rj < k && r0 + ri < n_rows ? x[(r0 + ri) * k + rj] : 0.f;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      float4 acc = zero4();
#pragma unroll
      for (int j = 0; j < KP; ++j) {
        const float v = __shfl_sync(0xffffffffu, xv, r * KP + j);
        acc = fma4(make_float4(v, v, v, v), wr[j], acc);
      }
      if (r0 + r < n_rows) st4(y + (r0 + r) * 128 + c, acc);
    }
  }
}

template <int KP>
__global__ void __launch_bounds__(RW_THREADS, KP == 8 ? 4 : 2)
k_small_linear_fwd(int64_t n_rows, int k, const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y) {
  pdl_sync();
  small_linear_fwd<KP>(n_rows, k, x, w, y);
}
__global__ void __launch_bounds__(RW_THREADS, 4) k_many_small_linears(int64_t n_rows, const __grid_constant__ ManyLinears a) {
  pdl_sync();
  small_linear_fwd<8>(n_rows, 7, a.x[blockIdx.y], a.w[blockIdx.y], a.y[blockIdx.y]);
}

// dx = dy W: every lane's 32 partial sums (32 / KP rows x KP) are reduced across the warp by halving, 31 shuffles in all, which leaves
// lane l with the sum number l = row * KP + j (reduced one by one they were 5 shuffles each).
template <int KP>
__global__ void __launch_bounds__(RW_THREADS, KP == 8 ? 3 : 2)
k_small_linear_bwd(int64_t n_rows, int k, const float* __restrict__ dy, const float* __restrict__ w, float* __restrict__ dx,
                   int accumulate) {
  constexpr int ROWS = 32 / KP;
  const int lane = threadIdx.x & 31, c = lane * 4, ri = lane / KP, rj = lane % KP;
  const int64_t step = ((int64_t)gridDim.x * blockDim.x >> 5) * ROWS;
  float4 wr[KP];
  pdl_sync();
  small_linear_weights<KP>(w, k, c, wr);
  for (int64_t r0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * ROWS; r0 < n_rows; r0 += step) {
    float4 g[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) g[r] = ld4(dy + (r0 + r < n_rows ? r0 + r : n_rows - 1) * 128 + c);
    const bool mine = rj < k && r0 + ri < n_rows;
    float* const out = dx + (r0 + ri) * k + rj;
    const float old = accumulate && mine ? *out : 0.f;
    float v[32];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int j = 0; j < KP; ++j) v[r * KP + j] = dot4(g[r], wr[j]);
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
      const bool upper = lane & h;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const float keep = upper ? v[i + h] : v[i], give = upper ? v[i] : v[i + h];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, h);
      }
    }
    if (mine) *out = v[0] + old;
  }
}

// ------------------------------------------------------------------ norms
__global__ void k_layernorm_fwd(int64_t n_rows, const float* __restrict__ x, const float* __restrict__ w,
                                const float* __restrict__ b, float* __restrict__ y) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float4 v = ld4(x + row * 128 + c);
  const float mean = warp_sum(v.x + v.y + v.z + v.w) * (1.f / 128.f);
  const float4 dv = make_float4(v.x - mean, v.y - mean, v.z - mean, v.w - mean);
  const float rstd = rsqrtf(warp_sum(dot4(dv, dv)) * (1.f / 128.f) + 1e-5f);
  st4(y + row * 128 + c, fma4(scl4(dv, rstd), ld4(w + c), ld4(b + c)));
}

__global__ void k_layernorm_bwd(int64_t n_rows, const float* __restrict__ x, const float* __restrict__ w,
                                const float* __restrict__ dy, float* __restrict__ dx) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float4 v = ld4(x + row * 128 + c);
  const float mean = warp_sum(v.x + v.y + v.z + v.w) * (1.f / 128.f);
  const float4 dv = make_float4(v.x - mean, v.y - mean, v.z - mean, v.w - mean);
  const float rstd = rsqrtf(warp_sum(dot4(dv, dv)) * (1.f / 128.f) + 1e-5f);
  const float4 xh = scl4(dv, rstd);
  const float4 g = mul4(ld4(dy + row * 128 + c), ld4(w + c));
  const float m1 = warp_sum(g.x + g.y + g.z + g.w) * (1.f / 128.f);
  const float m2 = warp_sum(dot4(g, xh)) * (1.f / 128.f);
  st4(dx + row * 128 + c, make_float4(rstd * (g.x - m1 - xh.x * m2), rstd * (g.y - m1 - xh.y * m2),
                                      rstd * (g.z - m1 - xh.z * m2), rstd * (g.w - m1 - xh.w * m2)));
}

__global__ void k_rmsnorm_fwd(int64_t n_rows, const float* __restrict__ x, const float* __restrict__ w,
                              float* __restrict__ y) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float4 v = ld4(x + row * 128 + c);
  const float r = rsqrtf(warp_sum(dot4(v, v)) * (1.f / 128.f) + RMS_EPS);
  st4(y + row * 128 + c, mul4(scl4(v, r), ld4(w + c)));
}

__global__ void k_rmsnorm_bwd(int64_t n_rows, const float* __restrict__ x, const float* __restrict__ w,
                              const float* __restrict__ dy, float* __restrict__ dx) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float4 v = ld4(x + row * 128 + c);
  const float r = rsqrtf(warp_sum(dot4(v, v)) * (1.f / 128.f) + RMS_EPS);
  const float4 n = scl4(v, r);
  const float4 g = mul4(ld4(dy + row * 128 + c), ld4(w + c));
  const float m = warp_sum(dot4(g, n)) * (1.f / 128.f);
  st4(dx + row * 128 + c, scl4(sub4(g, scl4(n, m)), r));
}

__global__ void k_embedding(int64_t n_rows, const int32_t* __restrict__ idx, int offset,
                            const float* __restrict__ table, float* __restrict__ y) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  st4(y + row * 128 + c, ld4(table + (int64_t)(idx[row] + offset) * 128 + c));
}

// ------------------------------------------------------------------ head projections
__global__ void k_head_dot_fwd(int64_t n_rows, int k, const float* __restrict__ z, const float* __restrict__ w,
                               const float* __restrict__ b, int take_abs, float* __restrict__ out) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  float s = 0.f;
  for (int j = c; j < k; j += 128) {
    const float4 v = ld4(z + row * k + j), ww = ld4(w + j);
    s += silu_f(v.x) * ww.x + silu_f(v.y) * ww.y + silu_f(v.z) * ww.z + silu_f(v.w) * ww.w;
  }
  s = warp_sum(s) + b[0];
  if (lane == 0) out[row] = take_abs ? fabsf(s) : s;
}

__global__ void k_head_dot_bwd(int64_t n_rows, int k, const float* __restrict__ z, const float* __restrict__ w,
                               const float* __restrict__ seed, const int32_t* __restrict__ seed_map,
                               float* __restrict__ dz) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float g = seed ? seed[seed_map ? seed_map[row] : row] : 1.f;
  for (int j = c; j < k; j += 128) {
    const float4 v = ld4(z + row * k + j), ww = ld4(w + j);
    st4(dz + row * k + j, make_float4(g * ww.x * silu_grad_f(v.x), g * ww.y * silu_grad_f(v.y),
                                      g * ww.z * silu_grad_f(v.z), g * ww.w * silu_grad_f(v.w)));
  }
}

__global__ void k_silu_bwd(int64_t n_rows, const float* __restrict__ dy, const float* __restrict__ z,
                           float* __restrict__ dz) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_rows)
  const float4 g = ld4(dy + row * 128 + c), v = ld4(z + row * 128 + c);
  st4(dz + row * 128 + c, make_float4(g.x * silu_grad_f(v.x), g.y * silu_grad_f(v.y), g.z * silu_grad_f(v.z),
                                      g.w * silu_grad_f(v.w)));
}

__global__ void k_segment_sum_scalar(int n_seg, const int32_t* __restrict__ seg_ptr, const float* __restrict__ x,
                                     float* __restrict__ out) {
  pdl_sync();
  MB_ROW_PROLOGUE(n_seg)
  float s = 0.f;
  for (int i = seg_ptr[row] + lane; i < seg_ptr[row + 1]; i += 32) s += x[i];
  s = warp_sum(s);
  if (lane == 0) out[row] = s;
}

}  // namespace mb

using namespace mb;
#define STREAM ((cudaStream_t)stream)
#define MB_REQUIRE(cond) do { if (!(cond)) return MB_ERR_INVALID; } while (0)

extern "C" int mb_gate_fwd(int64_t n_rows, const float* z, const float* w_core, const float* w_gate, float* h,
                           const float* res, const float* res_w, float* out2, void* stream) {
  MB_REQUIRE(n_rows >= 0 && z && w_core && w_gate && (h || out2) && (!out2 || res));
  if (n_rows == 0) return MB_OK;
  launch(k_gate_fwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, z, w_core, w_gate, h, res, res_w, out2);
  MB_LAUNCH_CHECK("k_gate_fwd");
  return MB_OK;
}

extern "C" int mb_gate_bwd(int64_t n_rows, const float* z, const float* w_core, const float* w_gate, const float* dh,
                           float* dz, void* stream) {
  MB_REQUIRE(n_rows >= 0 && z && w_core && w_gate && dh && dz);
  if (n_rows == 0) return MB_OK;
  launch(k_gate_bwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, z, w_core, w_gate, dh, dz);
  MB_LAUNCH_CHECK("k_gate_bwd");
  return MB_OK;
}

extern "C" int mb_seg_attn_fwd(int32_t n_nodes, const int32_t* tgt_ptr, const int32_t* src_ptr,
                               const int32_t* src_perm, const int32_t* emap, const float* logits, const float* h,
                               float* agg_t, float* agg_s, float* stats, void* stream) {
  MB_REQUIRE(n_nodes >= 0 && tgt_ptr && src_ptr && src_perm && logits && h && agg_t && agg_s && stats);
  if (n_nodes == 0) return MB_OK;
  // with an edge map the rows are directed edges and the nodes atoms: long segments
  if (emap)
    launch(k_seg_attn_fwd<4>, 2 * (unsigned)n_nodes, 128, 0, STREAM, n_nodes, tgt_ptr, src_ptr, src_perm, emap, logits, h, agg_t,
           agg_s, stats);
  else
    launch(k_seg_attn_fwd<1>, row_grid(2 * (int64_t)n_nodes), RW_THREADS, 0, STREAM, n_nodes, tgt_ptr, src_ptr, src_perm, emap,
           logits, h, agg_t, agg_s, stats);
  MB_LAUNCH_CHECK("k_seg_attn_fwd");
  return MB_OK;
}

extern "C" int mb_seg_attn_bwd(int64_t n_rows, const int32_t* tgt, const int32_t* src, int32_t idx_stride,
                               const int32_t* emap, const float* logits, const float* h, const float* agg_t,
                               const float* agg_s, const float* stats, const float* dagg_t, const float* dagg_s,
                               const float* dh_in, const int32_t* dh_map, float dh_scale, float* dh, float* dlogits,
                               const float* gate_z, const float* gate_wc, const float* gate_wg, float* gate_dz,
                               void* stream) {
  MB_REQUIRE(n_rows >= 0 && tgt && src && idx_stride > 0 && logits && h && agg_t && agg_s && stats && dagg_t &&
             dagg_s && dlogits && (gate_dz ? (gate_z && gate_wc && gate_wg) : dh != nullptr));
  if (n_rows == 0) return MB_OK;
  RowGrad a = {};
  a.idx_stride = idx_stride; a.dh_in = dh_in; a.dh_map = dh_map; a.dh_scale = dh_scale; a.tgt = tgt; a.src = src; a.emap = emap;
  a.logits = logits; a.h = h; a.agg_t = agg_t; a.agg_s = agg_s; a.stats = stats; a.dagg_t = dagg_t; a.dagg_s = dagg_s;
  a.dlogits = dlogits; a.z2 = gate_z; a.norm_core = gate_wc; a.norm_gate = gate_wg;
  launch(k_seg_attn_bwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, a, dh, gate_dz);
  MB_LAUNCH_CHECK("k_seg_attn_bwd");
  return MB_OK;
}

extern "C" int mb_seg_smooth_sum_fwd(int32_t n_nodes, const int32_t* tgt_ptr, const int32_t* emap,
                                     const int32_t* src, int32_t idx_stride, const float* env, const float* h,
                                     float* agg, void* stream) {
  MB_REQUIRE(n_nodes >= 0 && tgt_ptr && (emap || src) && env && h && agg && idx_stride > 0);
  if (n_nodes == 0) return MB_OK;
  if (!src)
    launch(k_seg_smooth_sum_fwd<8>, (unsigned)n_nodes, 256, 0, STREAM, n_nodes, tgt_ptr, emap, src, idx_stride, env, h, agg);
  else
    launch(k_seg_smooth_sum_fwd<1>, row_grid(n_nodes), RW_THREADS, 0, STREAM, n_nodes, tgt_ptr, emap, src, idx_stride, env, h,
           agg);
  MB_LAUNCH_CHECK("k_seg_smooth_sum_fwd");
  return MB_OK;
}

extern "C" int mb_seg_smooth_sum_bwd_rows(int64_t n_rows, const int32_t* tgt, const int32_t* src, int32_t idx_stride,
                                          const int32_t* emap, const float* env, const float* dagg, float* dh,
                                          int32_t accumulate, const float* gate_z, const float* gate_wc,
                                          const float* gate_wg, float* gate_dz, void* stream) {
  MB_REQUIRE(n_rows >= 0 && tgt && (emap || src) && env && dagg && idx_stride > 0 && (dh || (gate_dz && !accumulate)) &&
             (!gate_dz || (gate_z && gate_wc && gate_wg)));
  if (n_rows == 0) return MB_OK;
  RowGrad a = {};
  a.idx_stride = idx_stride; a.dh_in = accumulate ? dh : nullptr; a.tgt = tgt; a.src = src; a.emap = emap; a.env = env; a.dagg = dagg;
  a.z2 = gate_z; a.norm_core = gate_wc; a.norm_gate = gate_wg;
  launch(k_seg_smooth_sum_bwd_rows, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, a, dh, gate_dz);
  MB_LAUNCH_CHECK("k_seg_smooth_sum_bwd_rows");
  return MB_OK;
}

extern "C" int mb_seg_smooth_sum_bwd_env(int32_t n_nodes, const int32_t* tgt_ptr, const int32_t* src_ptr,
                                         const int32_t* src_perm, const int32_t* tgt, const int32_t* src,
                                         int32_t idx_stride, const int32_t* u2d, const int32_t* rev, const float* env,
                                         const float* h, const float* dagg, const float* drow, float* denv,
                                         void* stream) {
  MB_REQUIRE(n_nodes >= 0 && tgt && h && dagg && denv && idx_stride > 0);
  if (n_nodes == 0) return MB_OK;
  if (!src_ptr) {
    MB_REQUIRE(u2d && rev && idx_stride == 1);
    launch(k_smooth_env_bwd_atom, row_grid(n_nodes), RW_THREADS, 0, STREAM, n_nodes, u2d, rev, tgt, h, dagg, drow, denv);
  } else {
    MB_REQUIRE(tgt_ptr && src_perm && src && env && !drow);
    launch(k_smooth_env_bwd_line, row_grid(n_nodes), RW_THREADS, 0, STREAM, n_nodes, tgt_ptr, src_ptr, src_perm, tgt, src,
                                                                       idx_stride, env, h, dagg, denv);
  }
  MB_LAUNCH_CHECK("k_smooth_env_bwd");
  return MB_OK;
}

extern "C" int mb_mul_rows_gather(int64_t n_rows, const float* x, const float* s, const int32_t* idx, float* y,
                                  void* stream) {
  MB_REQUIRE(n_rows >= 0 && x && s && y);
  if (n_rows == 0) return MB_OK;
  launch(k_mul_rows_gather, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, x, s, idx, y);
  MB_LAUNCH_CHECK("k_mul_rows_gather");
  return MB_OK;
}

extern "C" int mb_seg_sum(int32_t n_nodes, int64_t n_rows, const int32_t* tgt_ptr, const int32_t* src_ptr,
                          const int32_t* src_perm, const int32_t* ctr, const float* x, float* out, float* ctr_out,
                          void* stream) {
  MB_REQUIRE(n_nodes >= 0 && n_rows >= 0 && tgt_ptr && src_ptr && src_perm && x && out && (!ctr || ctr_out));
  if (n_nodes == 0) return MB_OK;
  // long segments on average (and no per-centre sums, which follow the order of the rows): a block per segment and side
  if (!ctr && n_rows >= 16 * (int64_t)n_nodes)
    launch(k_seg_sum<8>, 2 * (unsigned)n_nodes, 256, 0, STREAM, n_nodes, tgt_ptr, src_ptr, src_perm, ctr, x, out, ctr_out);
  else
    launch(k_seg_sum<1>, row_grid(2 * (int64_t)n_nodes), RW_THREADS, 0, STREAM, n_nodes, tgt_ptr, src_ptr, src_perm, ctr, x, out,
                                                                           ctr_out);
  MB_LAUNCH_CHECK("k_seg_sum");
  return MB_OK;
}

extern "C" int mb_pair_sum(int32_t n_bonds, const int32_t* u2d, const int32_t* rev, const float* a, const float* b, float* out,
                           void* stream) {
  MB_REQUIRE(n_bonds >= 0 && u2d && rev && a && out);
  if (n_bonds == 0) return MB_OK;
  launch(k_pair_sum, row_grid(n_bonds), RW_THREADS, 0, STREAM, n_bonds, u2d, rev, a, b, out, b ? 512 : 256);
  MB_LAUNCH_CHECK("k_pair_sum");
  return MB_OK;
}

extern "C" int mb_pair_mean_res(int32_t n_bonds, const int32_t* u2d, const int32_t* rev, const float* y,
                                const float* res, const float* res_w, float* out, void* stream) {
  MB_REQUIRE(n_bonds >= 0 && u2d && rev && y && out);
  if (n_bonds == 0) return MB_OK;
  launch(k_pair_mean_res, row_grid(n_bonds), RW_THREADS, 0, STREAM, n_bonds, u2d, rev, y, res, res_w, out);
  MB_LAUNCH_CHECK("k_pair_mean_res");
  return MB_OK;
}

extern "C" int mb_scale_rows(int64_t n_rows, const float* x, const float* a, float* y, int32_t accumulate,
                             void* stream) {
  MB_REQUIRE(n_rows >= 0 && x && y);
  if (n_rows == 0) return MB_OK;
  launch(k_scale_rows, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, x, a, y, accumulate);
  MB_LAUNCH_CHECK("k_scale_rows");
  return MB_OK;
}

// a warp loads its weights once: no more blocks than are resident at a time, which walk the rows
static inline unsigned small_linear_grid(int64_t n_rows, int rows_per_warp, int resident) {
  const int64_t blocks = (n_rows + rows_per_warp * (RW_THREADS / 32) - 1) / (rows_per_warp * (RW_THREADS / 32));
  return (unsigned)(blocks < resident ? blocks : resident);
}

extern "C" int mb_small_linear_fwd(int64_t n_rows, int32_t k, const float* x, const float* w, float* y, void* stream) {
  MB_REQUIRE(n_rows >= 0 && k >= 1 && k <= 16 && x && w && y);
  if (n_rows == 0) return MB_OK;
  int n_sm = 0;
  if (const int rc = sm_count(&n_sm)) return rc;
  if (k <= 8) launch(k_small_linear_fwd<8>, small_linear_grid(n_rows, 4, 4 * n_sm), RW_THREADS, 0, STREAM, n_rows, k, x, w, y);
  else launch(k_small_linear_fwd<16>, small_linear_grid(n_rows, 2, 2 * n_sm), RW_THREADS, 0, STREAM, n_rows, k, x, w, y);
  MB_LAUNCH_CHECK("k_small_linear_fwd");
  return MB_OK;
}

extern "C" int mb_small_linear_bwd(int64_t n_rows, int32_t k, const float* dy, const float* w, float* dx,
                                   int32_t accumulate, void* stream) {
  MB_REQUIRE(n_rows >= 0 && k >= 1 && k <= 16 && dy && w && dx);
  if (n_rows == 0) return MB_OK;
  int n_sm = 0;
  if (const int rc = sm_count(&n_sm)) return rc;
  if (k <= 8)
    launch(k_small_linear_bwd<8>, small_linear_grid(n_rows, 4, 3 * n_sm), RW_THREADS, 0, STREAM, n_rows, k, dy, w, dx, accumulate);
  else
    launch(k_small_linear_bwd<16>, small_linear_grid(n_rows, 2, 2 * n_sm), RW_THREADS, 0, STREAM, n_rows, k, dy, w, dx, accumulate);
  MB_LAUNCH_CHECK("k_small_linear_bwd");
  return MB_OK;
}

extern "C" int mb_layernorm_fwd(int64_t n_rows, const float* x, const float* w, const float* b, float* y,
                                void* stream) {
  MB_REQUIRE(n_rows >= 0 && x && w && b && y);
  if (n_rows == 0) return MB_OK;
  launch(k_layernorm_fwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, x, w, b, y);
  MB_LAUNCH_CHECK("k_layernorm_fwd");
  return MB_OK;
}

extern "C" int mb_layernorm_bwd(int64_t n_rows, const float* x, const float* w, const float* dy, float* dx,
                                void* stream) {
  MB_REQUIRE(n_rows >= 0 && x && w && dy && dx);
  if (n_rows == 0) return MB_OK;
  launch(k_layernorm_bwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, x, w, dy, dx);
  MB_LAUNCH_CHECK("k_layernorm_bwd");
  return MB_OK;
}

extern "C" int mb_rmsnorm_fwd(int64_t n_rows, const float* x, const float* w, float* y, void* stream) {
  MB_REQUIRE(n_rows >= 0 && x && w && y);
  if (n_rows == 0) return MB_OK;
  launch(k_rmsnorm_fwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, x, w, y);
  MB_LAUNCH_CHECK("k_rmsnorm_fwd");
  return MB_OK;
}

extern "C" int mb_rmsnorm_bwd(int64_t n_rows, const float* x, const float* w, const float* dy, float* dx,
                              void* stream) {
  MB_REQUIRE(n_rows >= 0 && x && w && dy && dx);
  if (n_rows == 0) return MB_OK;
  launch(k_rmsnorm_bwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, x, w, dy, dx);
  MB_LAUNCH_CHECK("k_rmsnorm_bwd");
  return MB_OK;
}

extern "C" int mb_embedding(int64_t n_rows, const int32_t* idx, int32_t offset, const float* table, float* y,
                            void* stream) {
  MB_REQUIRE(n_rows >= 0 && idx && table && y);
  if (n_rows == 0) return MB_OK;
  launch(k_embedding, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, idx, offset, table, y);
  MB_LAUNCH_CHECK("k_embedding");
  return MB_OK;
}

extern "C" int mb_head_dot_fwd(int64_t n_rows, int32_t k, const float* z, const float* w, const float* b,
                               int32_t take_abs, float* out, void* stream) {
  MB_REQUIRE(n_rows >= 0 && k > 0 && (k % 128) == 0 && z && w && b && out);
  if (n_rows == 0) return MB_OK;
  launch(k_head_dot_fwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, k, z, w, b, take_abs, out);
  MB_LAUNCH_CHECK("k_head_dot_fwd");
  return MB_OK;
}

extern "C" int mb_head_dot_bwd(int64_t n_rows, int32_t k, const float* z, const float* w, const float* seed,
                               const int32_t* seed_map, float* dz, void* stream) {
  MB_REQUIRE(n_rows >= 0 && k > 0 && (k % 128) == 0 && z && w && dz);
  if (n_rows == 0) return MB_OK;
  launch(k_head_dot_bwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, k, z, w, seed, seed_map, dz);
  MB_LAUNCH_CHECK("k_head_dot_bwd");
  return MB_OK;
}

extern "C" int mb_silu_bwd(int64_t n_rows, const float* dy, const float* z, float* dz, void* stream) {
  MB_REQUIRE(n_rows >= 0 && dy && z && dz);
  if (n_rows == 0) return MB_OK;
  launch(k_silu_bwd, row_grid(n_rows), RW_THREADS, 0, STREAM, n_rows, dy, z, dz);
  MB_LAUNCH_CHECK("k_silu_bwd");
  return MB_OK;
}

extern "C" int mb_segment_sum_scalar(int32_t n_seg, const int32_t* seg_ptr, const float* x, float* out,
                                     void* stream) {
  MB_REQUIRE(n_seg >= 0 && seg_ptr && x && out);
  if (n_seg == 0) return MB_OK;
  launch(k_segment_sum_scalar, row_grid(n_seg), RW_THREADS, 0, STREAM, n_seg, seg_ptr, x, out);
  MB_LAUNCH_CHECK("k_segment_sum_scalar");
  return MB_OK;
}

namespace mb {
int many_small_linears(int64_t n_rows, int n, const ManyLinears& a, cudaStream_t stream) {
  if (n_rows == 0 || n == 0) return MB_OK;
  int n_sm = 0;
  if (const int rc = sm_count(&n_sm)) return rc;
  launch(k_many_small_linears, dim3(small_linear_grid(n_rows, 4, 4 * n_sm), (unsigned)n), RW_THREADS, 0, stream, n_rows, a);
  MB_LAUNCH_CHECK("k_many_small_linears");
  return MB_OK;
}
int smooth_env_bwd_rbf(int32_t n_bonds, const mb_row_graph& g, const float* env, const float* h, const float* dagg, const float* drow,
                       const float* w, float* d_rbf, cudaStream_t stream) {
  if (n_bonds == 0) return MB_OK;
  if (g.is_atom)
    launch(k_smooth_env_bwd_atom_rbf, row_grid(n_bonds), RW_THREADS, 0, stream, n_bonds, g.u2d, g.rev, g.tgt, h, dagg, drow, w, d_rbf);
  else
    launch(k_smooth_env_bwd_line_rbf, row_grid(n_bonds), RW_THREADS, 0, stream, n_bonds, g.tgt_ptr, g.src_ptr, g.src_perm, g.tgt,
           g.src, env, h, dagg, w, d_rbf);
  MB_LAUNCH_CHECK("k_smooth_env_bwd_rbf");
  return MB_OK;
}
}  // namespace mb
