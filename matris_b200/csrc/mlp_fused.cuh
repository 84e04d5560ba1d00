// Fused two-layer row MLPs, forward and backward (included by gemm.cu inside namespace mb, after gemm_persistent.cuh).
//
//   GATED_FWD  z1 = X W1^T + b1 + sum_i T_i[idx_i]      [rows, 256] = core | gate      X: up to four gathered 128-wide segments
//              z2 = SiLU(z1) W2^T + b2 per branch       h = SiLU(RMSNorm(z2_core) w_c) * sigmoid(RMSNorm(z2_gate) w_g)
//   PLAIN_FWD  z1 = X W1^T + b1,  y = SiLU(z1) W2^T + b2                               [rows, 128]
//   GATED_BWD  dz1 = (dz2 W2 per branch) * SiLU'(z1),  dx = dz1 W1e + E W3            dx: the gradient of ONE 128-wide segment
//   PLAIN_BWD  dz1 = scale (dy W2) * SiLU'(z1),  dx = dz1 W1
//   each with the optional second output out2 = result + res_w * res.
//
// The addends T_i are tables of node terms: the part of layer 1 that belongs to a gathered segment, W1_seg node, is the same
// for every row that gathers the node, so it is formed once per node (a GEMM over nodes) and gathered here as 256 finished
// sums instead of 128 operands.  A triplet row then contracts K = 128 instead of 384 or 512.
//
// 3xBF16 arithmetic as in gemm_persistent.cuh.  One persistent CTA per SM, 128-row tiles, tcgen05 throughout:
//
//   L1    A (32-float K chunks, gathered, split into bf16 hi / lo, in four tensor-memory buffers; a chunk feeds both branches)
//         x W1 -> accumulator regions (128 x 128 fp32)
//   mid   four epilogue warps per region read it (thread = row), add the addends / multiply by SiLU'(z1), apply SiLU, split and
//         write the result back IN PLACE as the bf16 A operand of layer 2: 32 fp32 columns become 16 hi + 16 lo columns
//   L2    A = that region, x W2 -> a region that is free
//   epi   RMSNorm, activations, residual, output
//
// What bounds it is HBM (for 573,894 triplet rows with z1 / z2 kept: 3.5 KB per row = 0.31 ms at the copy rate) provided that
// nothing queues in front of it.  Rows move by TMA in both directions (32 rows x 32 floats per copy, 128-byte swizzle, so that a
// thread reads or writes its row in 16-byte pieces without bank conflicts): through registers and st.global every 4 KB cost 64
// more wavefronts of the L1 pipe, and a warp's shared-memory accesses and barrier polls waited behind its own stores.  Only
// gathered rows (addend tables, indexed sources) are loaded by the producer warps themselves, eight lanes per 128-byte line.
//
// Regions (three of 128 columns from 0; A buffers from 384).  GATED_FWD rotates: tile t (r = t mod 3) has L1 core -> r, L1 gate
// -> r+1, L2 core -> r+2, L2 gate -> r (its A operand, the core's activations, has been consumed).  Tile t+1's core starts in
// r+1 as soon as L2 gate(t) is done, under the epilogue of t.  GATED_BWD: 0, 1 and 2.  PLAIN_*: tiles alternate between the
// two epilogue groups, L1(t) -> 2t mod 3, L2(t) -> 2t+1 mod 3, issued L1(t+1) before L2(t).
//
// Measured behind an L2 flush (bench_gemm.py; addend tables of a fifth of the rows), 573,894 rows with z1 and z2 kept: two
// addends and a residual 0.49 ms, three addends 0.53 (nothing kept: 0.40), no contraction and three addends 0.48, K = 384
// gathered with a residual 0.63; GATED_BWD with a residual 0.42, with E too 0.59; FFN forward 0.22, backward 0.17.  The smallest
// launches that k_few leaves (9,473 rows: one tile for half of the multiprocessors) are bound by the chain of a tile's stages:
// back to back 19.0 us for the gated forward with two addends, 22.5 with K = 384, 13.5 for its backward, 17.2 with E, 12.0 for
// the FFN, 9.2 for its backward.  The epilogues' arithmetic goes two values at a time (f2, common.cuh); 523,000 rows: three
// addends 0.497 -> 0.483 (nothing kept 0.382 -> 0.364), no contraction 0.439 -> 0.433, FFN forward 0.208 -> 0.202, backward
// 0.169 -> 0.156.  (The addends' own sums that way: 0.523.)  With three addends 44 % of the cycles issue an instruction, the
// load / store data pipe is busy in 44 %, the tensor pipe in 20 %: 4.5 warps a scheduler wait for their own chains.
//
// Warps: 0 MMA, 1 TMA (weights, 16 KB tiles of 64 K values, five slots), 2-9 producers, 10-17 epilogue (two groups of four; the
// group's branch or tile parity, the warp's lane quarter).  Every mbarrier wait is bounded; on expiry the status word is set, the
// role stops waiting and runs to the common exit.  Every waiter sees every phase of a barrier it waits on.

enum MlpMode { MLP_GATED_FWD = 0, MLP_PLAIN_FWD = 1, MLP_GATED_BWD = 2, MLP_PLAIN_BWD = 3 };

struct MlpArgs {
  int64_t n_rows;
  int32_t n_src, n_ext, n_add, pad;
  mb_src src[4];             // A of layer 1 (GATED_BWD: core and gate half of dz2)
  mb_src ext[2];             // GATED_BWD: further A segments of the second contraction (E)
  mb_add add[3];             // GATED_FWD: addends
  const float* side;         // *_BWD: z1
  int64_t ld_side;
  const float *b1, *b2, *norm_core, *norm_gate;
  float* z1; int64_t ld_z1;  // *_FWD: z1, GATED_BWD: dz1 (optional)
  float* z2; int64_t ld_z2;
  float* h; int64_t ld_h;
  const float* res; const float* res_w; int64_t ld_res;
  float* out2; int64_t ld_out2;
  float scale;               // PLAIN_BWD
};
struct alignas(64) MlpMaps {
  CUtensorMap w1[2], w2[2], w3[2];       // weights: hi, lo; boxes of 128 rows x 64 values
  CUtensorMap src[4], ext[2], side, res; // rows read in place; boxes of 32 rows x 32 floats
  CUtensorMap z1, z2, h, out2;           // rows written
};

constexpr int ML_THREADS = 576;
constexpr int ML_MMA_WARP = 0, ML_TMA_WARP = 1, ML_PROD_WARP0 = 2, ML_EPI_WARP0 = 10;
constexpr uint32_t ML_W_SLOTS = 5;
constexpr uint32_t ML_A_BASE = 384;
constexpr int ML_PATCH = 32 * 128;                             // 32 rows x 32 floats
constexpr int ML_CONV_OFF = ML_W_SLOTS * TC_TILE_BYTES;        // one patch per producer warp
constexpr int ML_SIDE_OFF = ML_CONV_OFF + 8 * ML_PATCH;        // two per epilogue warp, filled by its producer warp
constexpr int ML_STAGE_OFF = ML_SIDE_OFF + 16 * ML_PATCH;      // one per epilogue warp
constexpr int ML_CONST_OFF = ML_STAGE_OFF + 8 * ML_PATCH;      // b1[256] b2[256] norm_core[128] norm_gate[128] res_w[128]
constexpr int ML_RINV_OFF = ML_CONST_OFF + 896 * 4;            // [tile parity][branch][row]
constexpr int ML_BAR_OFF = ML_RINV_OFF + 2 * 2 * 128 * 4;
constexpr int ML_SMEM_BYTES = ML_BAR_OFF + 640;
constexpr float ML_RMS_EPS = 1.1920928955078125e-07f;          // nn.RMSNorm(eps=None): float32 machine epsilon
static_assert(ML_SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ void sts4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ float4 lds4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// Between ordinary accesses of a patch and the copy engine's writes to it: a barrier orders the threads, not the two proxies.
// Any thread on the path from the last ordinary store to the copy may execute it; here it is the one that issues the copy.
__device__ __forceinline__ void to_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 32 row values (thread = row) <-> the swizzled patch: 16-byte chunk j of row r sits at position j ^ (r & 7)
__device__ __forceinline__ void patch_put(uint32_t patch, int lane, const float (&x)[32]) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
    sts4(patch + lane * 128 + ((j ^ (lane & 7)) << 4), x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
}
// patch -> rows y.., columns x.. of a tensor (rows past its end are not written)
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t patch, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               :: "l"(reinterpret_cast<uint64_t>(map)), "r"(patch), "r"(x), "r"(y) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// rows y.., columns x.. of a tensor -> patch (one lane)
__device__ __forceinline__ void load_patch(const CUtensorMap* map, uint32_t patch, uint32_t bar, int x, int y) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(ML_PATCH) : "memory");
  tma_load_2d(patch, map, bar, x, y);
}
__device__ __forceinline__ void tmem_get(uint32_t addr, float (&x)[32]) {
  uint32_t v[32];
  MB_TMEM_LD32(addr, v);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(v[i]);
}

// SiLU(a) sigmoid(b) = a / ((1 + e^-a) (1 + e^-b)): one reciprocal for both (the special-function pipe, a quarter of the rate of
// the others, bounds this pass)
__device__ __forceinline__ float gated_value(float a, float b) {
  float ea, eb, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ea) : "f"(a * -1.442695041f));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(eb) : "f"(b * -1.442695041f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"((1.0f + ea) * (1.0f + eb)));
  return a * r;
}
__device__ __forceinline__ f2 gated_value(f2 a, f2 b) {
  const f2 c = two(-1.442695041f, -1.442695041f), one = two(1.f, 1.f);
  float a0, a1, b0, b1;
  apart(a * c, a0, a1);
  apart(b * c, b0, b1);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a0));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a1));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(b0));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(b1));
  apart((one + two(a0, a1)) * (one + two(b0, b1)), a0, a1);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(a0));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(a1));
  return a * two(a0, a1);
}

// Sum of squares of 32 values of a row, halves added to halves: the order in which k_few adds them across its lanes, so that a row's
// norm does not depend on which kernel a launch of its size takes.
__device__ __forceinline__ float sum_of_squares(const float (&y)[32]) {
  float v[16];
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    const f2 lower = two(y[i], y[i + 1]), upper = two(y[i + 16], y[i + 17]);
    apart(fma2(upper, upper, lower * lower), v[i], v[i + 1]);
  }
#pragma unroll
  for (int n = 8; n > 1; n >>= 1)
#pragma unroll
    for (int i = 0; i < n; i += 2) apart(two(v[i], v[i + 1]) + two(v[i + n], v[i + n + 1]), v[i], v[i + 1]);
  return v[0] + v[1];
}

// N_ADD: GATED_FWD's number of addends (a launch without any keeps the registers of their gather)
template <int MODE, int N_ADD = 0>
__global__ void __launch_bounds__(ML_THREADS, 1)
k_mlp(const __grid_constant__ MlpArgs d, const __grid_constant__ MlpMaps maps) {
  constexpr bool GATED = MODE == MLP_GATED_FWD || MODE == MLP_GATED_BWD;
  // Who asks for the residual's patches, which follow a tile's side patches in the same two buffers.  GATED_FWD: the epilogue warp
  // itself when it is done with what a buffer held; left to the producer, whose addends are a latency-bound gather, the chunks of
  // the next tile wait for that (0.65 against 0.59 ms for 573,894 rows).  The others: the producer (their epilogue is the busier side:
  // 0.61 against 0.62 ms backward).
  constexpr bool EPI_RES = MODE == MLP_GATED_FWD;
  constexpr bool FWD = MODE == MLP_GATED_FWD || MODE == MLP_PLAIN_FWD;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ML_BAR_OFF);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + ML_BAR_OFF + 632);
  const uint32_t sm0 = smem_u32(smem);
  if ((sm0 & 1023u) != 0) {  // the swizzled tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicOr(&g_gemm_status, 2);
    return;
  }
  // a_ready[4] (4 producer warps) a_done[4] | w_ready[5] w_done[5] | d1_full[2] (L1 of branch / group) | d2_full[2] (L2) |
  // mid_ready[2][4] (4 epilogue warps) | epi_done[2] | side_full[8][2] side_empty[8][2] | conv_full[8] | retired
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t a_ready = bar0, a_done = bar0 + 32, w_ready = bar0 + 64, w_done = bar0 + 104, d1_full = bar0 + 144,
                 d2_full = bar0 + 160, mid_ready = bar0 + 176, epi_done = bar0 + 240, side_full = bar0 + 256,
                 side_empty = bar0 + 384, conv_full = bar0 + 512, retired = bar0 + 576;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* const cst = reinterpret_cast<float*>(smem + ML_CONST_OFF);
  const int64_t n_rows = d.n_rows;
  const int n_row_tiles = (int)((n_rows + 127) >> 7);
  const int first_rt = (int)blockIdx.x, step_rt = (int)gridDim.x;
  const int n_tiles = (n_row_tiles - first_rt + step_rt - 1) / step_rt;  // the grid never exceeds the tile count
  const int n_kp1 = 2 * d.n_src, n_kpx = MODE == MLP_GATED_BWD ? 2 * d.n_ext : 0;  // pairs of 32-float K chunks
  const int n_kpa = n_kp1 + n_kpx;
  constexpr bool has_side = MODE == MLP_GATED_FWD ? N_ADD > 0 : !FWD;
  const bool has_res = d.out2 != nullptr;

  if (warp == ML_MMA_WARP) {
    if (lane == 0) {
      for (int b = 0; b < 4; ++b) { mbar_init(a_ready + 8 * b, 4); mbar_init(a_done + 8 * b, 1); }
      for (uint32_t b = 0; b < ML_W_SLOTS; ++b) { mbar_init(w_ready + 8 * b, 1); mbar_init(w_done + 8 * b, 1); }
      for (int b = 0; b < 2; ++b) {
        mbar_init(d1_full + 8 * b, 1); mbar_init(d2_full + 8 * b, 1); mbar_init(epi_done + 8 * b, GATED ? 8 : 4);
      }
      for (int b = 0; b < 8; ++b) { mbar_init(mid_ready + 8 * b, 4); mbar_init(conv_full + 8 * b, 1); }
      for (int b = 0; b < 16; ++b) { mbar_init(side_full + 8 * b, 1); mbar_init(side_empty + 8 * b, 1); }
      mbar_init(retired, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(tmem_slot)), "r"(PS_TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  // The sequence of K-chunk pairs both issuing warps walk: step(tile, kind, branch, pair)
  enum { L1 = 0, L2 = 1, EX = 2, L1_NONE = 3 };
  auto walk = [&](auto step) {
    if constexpr (GATED) {
      for (int t = 0; t < n_tiles; ++t) {
        if constexpr (FWD) {
          if (n_kp1 == 0) { step(t, L1_NONE, 0, 0); step(t, L1_NONE, 1, 0); }
          else if (n_kp1 <= 2) {  // all chunks of the tile are resident: the core branch need not wait for the gate's region
            for (int br = 0; br < 2; ++br)
              for (int kp = 0; kp < n_kp1; ++kp) step(t, L1, br, kp);
          } else {
            for (int kp = 0; kp < n_kp1; ++kp)
              for (int br = 0; br < 2; ++br) step(t, L1, br, kp);
          }
        } else {
          for (int br = 0; br < 2; ++br)
            for (int kp = 0; kp < 2; ++kp) step(t, L1, br, kp);
          for (int kp = 0; kp < n_kpx; ++kp) step(t, EX, 0, kp);
        }
        for (int br = 0; br < 2; ++br)
          for (int kp = 0; kp < 2; ++kp) step(t, L2, br, kp);
      }
    } else {
      for (int t = 0; t <= n_tiles; ++t) {
        if (t < n_tiles)
          for (int kp = 0; kp < n_kp1; ++kp) step(t, L1, 0, kp);
        if (t > 0)
          for (int kp = 0; kp < 2; ++kp) step(t - 1, L2, 0, kp);
      }
    }
  };

  if (warp == ML_MMA_WARP) {
    // ---------------------------------------------------------------- MMA warp (warp-uniform, one elected lane issues)
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t ring_u = __shfl_sync(0xffffffffu, sm0, 0);
    bool alive = true;
    uint32_t wslot = 0, wphase = 0;  // slot and phase of the next W tile
    auto wait = [&](uint32_t bar, uint32_t parity) { if (alive) alive = mbar_wait(bar, parity & 1); };
    walk([&](int t, int kind, int br, int kp) {
      const int g = GATED ? br : (t & 1);          // barrier set of the branch / of the tile's group
      const uint32_t par = (uint32_t)(GATED ? t : t >> 1);
      uint32_t a_reg, d_reg;
      bool fresh = kp == 0;
      if constexpr (MODE == MLP_GATED_FWD) {
        const uint32_t r = (uint32_t)t % 3u;
        if (kind == L1 || kind == L1_NONE) d_reg = (r + br) % 3u;
        else d_reg = br == 0 ? (r + 2) % 3u : r;
        a_reg = (r + br) % 3u;
        if (kp == 0) {
          if (kind != L2) {
            // core: the region was the A operand of the previous tile's last contraction; gate: its core result
            if (t > 0) { if (br == 0) wait(d2_full + 8, (uint32_t)(t - 1)); else wait(epi_done, (uint32_t)(t - 1)); }
          } else if (br == 1) {
            wait(d2_full, par);  // the result replaces the core's A operand
          }
        }
      } else if constexpr (MODE == MLP_GATED_BWD) {
        d_reg = kind == L1 ? (uint32_t)br : 2u;
        a_reg = (uint32_t)br;
        if (kind == L2 && (br == 1 || n_kpx > 0)) fresh = false;
        if (kp == 0 && t > 0) {
          if (kind == L1 && br == 0) wait(d2_full, (uint32_t)(t - 1));
          if (fresh && kind != L1) wait(epi_done, (uint32_t)(t - 1));
        }
      } else {
        a_reg = (uint32_t)(2 * t) % 3u;
        d_reg = kind == L1 ? a_reg : (uint32_t)(2 * t + 1) % 3u;
        if (kp == 0) {
          if (kind == L1) { if (t >= 2) wait(epi_done + 8 * (t & 1), (uint32_t)((t - 2) >> 1)); }
          else if (t >= 1) wait(d2_full + 8 * ((t - 1) & 1), (uint32_t)((t - 1) >> 1));
        }
      }
      if (kind == L1_NONE) {  // nothing to contract: the region may be written
        alive = __all_sync(0xffffffffu, alive);
        if (elected) mma_commit(d1_full + 8 * g);
        __syncwarp();
        return;
      }
      uint32_t ta, abuf = 0;
      if (kind == L2) {
        wait(mid_ready + 8 * (4 * g + 2 * kp), par);
        wait(mid_ready + 8 * (4 * g + 2 * kp + 1), par);
        ta = tmem_u + 128u * a_reg + 64u * (uint32_t)kp;
      } else {
        const int pair = kind == EX ? n_kp1 + kp : (MODE == MLP_GATED_BWD ? 2 * br + kp : kp);
        const uint32_t gp = (uint32_t)(t * n_kpa + pair);
        abuf = 2 * (gp & 1);
        wait(a_ready + 8 * abuf, gp >> 1);
        wait(a_ready + 8 * (abuf + 1), gp >> 1);
        ta = tmem_u + ML_A_BASE + 32u * abuf;
      }
      const uint32_t s_hi = wslot, p_hi = wphase;
      uint32_t s_lo = wslot + 1, p_lo = wphase;
      if (s_lo == ML_W_SLOTS) { s_lo = 0; ++p_lo; }
      wslot = s_lo + 1; wphase = p_lo;
      if (wslot == ML_W_SLOTS) { wslot = 0; ++wphase; }
      wait(w_ready + 8 * s_hi, p_hi);
      wait(w_ready + 8 * s_lo, p_lo);
      alive = __all_sync(0xffffffffu, alive);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d_tmem = tmem_u + 128u * d_reg;
      const bool a_last = kind != L2 && (MODE != MLP_GATED_FWD || br == 1);  // this A pair's last reader
      const int last_kp = kind == L2 || MODE == MLP_GATED_BWD ? 1 : n_kp1 - 1;
      if (elected) {
        const uint64_t dbh = umma_desc(ring_u + s_hi * TC_TILE_BYTES), dbl = umma_desc(ring_u + s_lo * TC_TILE_BYTES);
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {  // K steps of 16: 8 TMEM columns of A, 32 bytes (>> 4 = 2) of the W rows
            const uint64_t adv = (uint64_t)(2 * (2 * ch + kk));
            const uint32_t t_hi = ta + 32 * ch + 8 * kk, t_lo = t_hi + 16;
            umma_bf16_ts(d_tmem, t_lo, dbh + adv, (!fresh || ch > 0 || kk > 0) ? 1u : 0u);
            umma_bf16_ts(d_tmem, t_hi, dbl + adv, 1u);
            umma_bf16_ts(d_tmem, t_hi, dbh + adv, 1u);
          }
        }
        mma_commit(w_done + 8 * s_hi);
        mma_commit(w_done + 8 * s_lo);
        if (a_last) { mma_commit(a_done + 8 * abuf); mma_commit(a_done + 8 * (abuf + 1)); }
        if (kp == last_kp) {
          if (kind == L1) mma_commit(d1_full + 8 * g);
          if (kind == L2) {
            if constexpr (MODE == MLP_GATED_BWD) { if (br == 1) mma_commit(d2_full); }
            else mma_commit(d2_full + 8 * g);
          }
        }
      }
      __syncwarp();
    });
    drain_mma(retired, elected);
  } else if (warp == ML_TMA_WARP) {
    // ---------------------------------------------------------------- TMA warp: weight tiles, up to five ahead
    pdl_sync();
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    const uint32_t ring_u = __shfl_sync(0xffffffffu, sm0, 0);
    bool alive = true;
    uint32_t n = 0, slot = 0, phase = 0;
    walk([&](int t, int kind, int br, int kp) {
      if (kind == L1_NONE || !alive) return;
      const CUtensorMap* m = kind == L1 ? maps.w1 : kind == L2 ? maps.w2 : maps.w3;
      int x = 64 * kp, y = GATED ? 128 * br : 0;
      if constexpr (MODE == MLP_GATED_BWD) {
        if (kind == L2) { x = 128 * br + 64 * kp; y = 0; }
        if (kind == EX) y = 0;
      }
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        if (n >= ML_W_SLOTS && alive) alive = mbar_wait(w_done + 8 * slot, (phase - 1) & 1);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) return;
        if (elected) {
          const uint32_t bar = w_ready + 8 * slot;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(TC_TILE_BYTES) : "memory");
          tma_load_2d(ring_u + slot * TC_TILE_BYTES, m + part, bar, x, y);
        }
        __syncwarp();
        ++n;
        if (++slot == ML_W_SLOTS) { slot = 0; ++phase; }
      }
    });
    drain_copies(w_ready, ML_W_SLOTS, n);
  } else if (warp >= ML_EPI_WARP0) {
    // ---------------------------------------------------------------- epilogue warps
    pdl_sync();  // (the MMA warp touches nothing but this CTA's own memory)
    for (int i = tid - 32 * ML_EPI_WARP0; i < 896; i += 256) {
      float v = 0.f;
      if (i < 256) { if (FWD && d.b1 && (GATED || i < 128)) v = d.b1[i]; }
      else if (i < 512) { if (FWD && d.b2 && (GATED || i < 384)) v = d.b2[i - 256]; }
      else if (i < 768) { if (FWD && GATED) v = i < 640 ? d.norm_core[i - 512] : d.norm_gate[i - 640]; }
      else v = d.res_w ? d.res_w[i - 768] : 1.f;
      cst[i] = v;
    }
    asm volatile("bar.sync 5, 512;" ::: "memory");  // the constants are there: epilogue and producer warps
    const int e = warp - ML_EPI_WARP0, q = warp & 3, grp = e >> 2;
    const uint32_t lane_q = tmem_base + ((uint32_t)(q * 32) << 16);
    const uint32_t side0 = sm0 + ML_SIDE_OFF + e * 2 * ML_PATCH, stage = sm0 + ML_STAGE_OFF + e * ML_PATCH;
    const uint32_t my_full = side_full + 16 * e, my_empty = side_empty + 16 * e;
    const int br = GATED ? grp : 0;
    const float4* const b1s = reinterpret_cast<const float4*>(cst) + 32 * br;
    float* const rinvs = reinterpret_cast<float*>(smem + ML_RINV_OFF);
    bool alive = true;
    uint32_t side_n = 0;
    auto wait = [&](uint32_t bar, uint32_t parity) {
      if (alive) alive = mbar_wait(bar, parity & 1);
      alive = __all_sync(0xffffffffu, alive);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    // the warp's 32 x 32 values (thread = row) -> columns x.. of an output, through the staging patch
    auto write = [&](const CUtensorMap* map, const float (&v)[32], int x, int row0) {
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the previous copy has left the patch
      __syncwarp();
      patch_put(stage, lane, v);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0 && alive && row0 < n_rows) tma_store_2d(map, stage, x, row0);
    };
    uint32_t asked = 0;  // number after that of the last copy asked for
    auto request = [&](uint32_t n, int k, int row0) {  // residual patch k (EPI_RES)
      if (!alive) return;
      asked = n + 1;
      if (lane == 0) {
        to_async_proxy();  // the buffer held addend sums that a producer warp stored
        load_patch(&maps.res, side0 + (n & 1) * ML_PATCH, my_full + 8 * (n & 1), 64 * grp + 32 * k, row0);
      }
    };
    // finished columns `col`..: h = v and / or out2 = v + res_w * res (the residual rows arrive as a side patch)
    auto finish = [&](float (&v)[32], int col, int row0) {
      if (d.h) write(&maps.h, v, col, row0);
      if (has_res) {
        const uint32_t patch = side0 + (side_n & 1) * ML_PATCH;
        wait(my_full + 8 * (side_n & 1), side_n >> 1);
        const float4* const rws = reinterpret_cast<const float4*>(cst + 768 + col);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 x = lds4(patch + lane * 128 + ((j ^ (lane & 7)) << 4)), w = rws[j];
          fma4_to(v + 4 * j, x, w);
        }
        __syncwarp();
        if ((has_side || !EPI_RES) && lane == 0) mbar_arrive(my_empty + 8 * (side_n & 1));
        ++side_n;
        write(&maps.out2, v, col, row0);
      }
    };
    for (int t = GATED ? 0 : grp; t < n_tiles; t += GATED ? 1 : 2) {
      const uint32_t par = (uint32_t)(GATED ? t : t >> 1);
      const int row0 = (first_rt + t * step_rt) * 128 + q * 32;
      uint32_t reg_a, reg_d;  // region of L1 / the A operand, region of the result
      if constexpr (MODE == MLP_GATED_FWD) {
        const uint32_t r = (uint32_t)t % 3u;
        reg_a = (r + grp) % 3u;
        reg_d = grp == 0 ? (r + 2) % 3u : r;
      } else if constexpr (MODE == MLP_GATED_BWD) {
        reg_a = (uint32_t)grp;
        reg_d = 2;
      } else {
        reg_a = (uint32_t)(2 * t) % 3u;
        reg_d = (uint32_t)(2 * t + 1) % 3u;
      }
      if (EPI_RES && has_res && !has_side) {
        request(side_n, 0, row0);
        request(side_n + 1, 1, row0);
      }
      // ------------------------------------------------ mid
      wait(d1_full + 8 * grp, par);
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        const uint32_t ta = lane_q + 128u * reg_a + 32u * c;
        const uint32_t patch = side0 + (side_n & 1) * ML_PATCH;
        float x[32];
        if (!FWD || n_kp1 > 0) {
          tmem_get(ta, x);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] = 0.f;
        }
        if (has_side) wait(my_full + 8 * (side_n & 1), side_n >> 1);
        if constexpr (FWD) {
          if (has_side) {  // the addends' sum (b1 included)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 v = lds4(patch + lane * 128 + ((j ^ (lane & 7)) << 4));
              add4_to(x + 4 * j, v);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 v = b1s[8 * c + j];
              add4_to(x + 4 * j, v);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = lds4(patch + lane * 128 + ((j ^ (lane & 7)) << 4));
            if constexpr (MODE == MLP_PLAIN_BWD) {
              const f2 s = two(d.scale, d.scale);
              apart(two(x[4 * j], x[4 * j + 1]) * (s * silu_grad_fast_2(low(v))), x[4 * j], x[4 * j + 1]);
              apart(two(x[4 * j + 2], x[4 * j + 3]) * (s * silu_grad_fast_2(high(v))), x[4 * j + 2], x[4 * j + 3]);
            } else {
              silu_grad4_to(x + 4 * j, v);
            }
          }
        }
        if (has_side) {
          if (!EPI_RES || c < 2 || !has_res) {  // the side patch goes back to its producer
            __syncwarp();
            if (lane == 0) mbar_arrive(my_empty + 8 * (side_n & 1));
          }
          ++side_n;
        }
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          float sx[16];
          if constexpr (FWD) {
            silu_fast_all(x + 16 * hh, sx);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) sx[i] = x[16 * hh + i];
          }
          uint32_t hi[8], lo[8];
          split_bf16(sx, hi, lo);
          MB_TMEM_ST8(ta + 8 * hh, hi);
          MB_TMEM_ST8(ta + 16 + 8 * hh, lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(mid_ready + 8 * (4 * grp + c));
        if (EPI_RES && has_side && has_res && c >= 2) request(side_n + 1, c - 2, row0);
        if (d.z1) write(&maps.z1, x, 128 * br + 32 * c, row0);
      }
      if constexpr (MODE == MLP_GATED_FWD) {
        // ---------------------------------------------- pass 1: + b2, optional z2, sum of squares
        wait(d2_full + 8 * grp, par);
        const float4* const b2s = reinterpret_cast<const float4*>(cst + 256);
        const uint32_t own = lane_q + 128u * reg_d;
        float s01 = 0.f, s23 = 0.f;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          float y[32];
          tmem_get(own + 32u * c, y);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = b2s[32 * grp + 8 * c + j];
            add4_to(y + 4 * j, v);
          }
          const float s = sum_of_squares(y);
          if (c < 2) s01 += s;
          else s23 += s;
          if (d.z2) write(&maps.z2, y, 128 * grp + 32 * c, row0);
        }
        rinvs[((t & 1) * 2 + grp) * 128 + q * 32 + lane] = rsqrtf((s01 + s23) * (1.0f / 128.0f) + ML_RMS_EPS);
        wait(d2_full + 8 * (grp ^ 1), par);
        asm volatile("bar.sync %0, 64;" :: "r"(1 + q) : "memory");  // the two groups' warps of this lane quarter
        const float rc = rinvs[((t & 1) * 2) * 128 + q * 32 + lane], rg = rinvs[((t & 1) * 2 + 1) * 128 + q * 32 + lane];
        // ---------------------------------------------- pass 2: this group's 64 columns of both branches
        const f2 rc2 = two(rc, rc), rg2 = two(rg, rg);
        const float4* const nws = reinterpret_cast<const float4*>(cst + 512);
        const uint32_t r3 = (uint32_t)t % 3u;
        const uint32_t core = lane_q + 128u * ((r3 + 2) % 3u) + 64u * grp, gate = lane_q + 128u * r3 + 64u * grp;
#pragma unroll 1
        for (int j2 = 0; j2 < 2; ++j2) {
          const int c4 = 16 * grp + 8 * j2;  // float4 index of the first column
          float y[32];
          tmem_get(core + 32u * j2, y);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 bc = b2s[c4 + j], nc = nws[c4 + j];
            apart((two(y[4 * j], y[4 * j + 1]) + low(bc)) * (rc2 * low(nc)), y[4 * j], y[4 * j + 1]);
            apart((two(y[4 * j + 2], y[4 * j + 3]) + high(bc)) * (rc2 * high(nc)), y[4 * j + 2], y[4 * j + 3]);
          }
          float z[32];
          tmem_get(gate + 32u * j2, z);
          if (j2 == 1) {  // both results have been read for the last time
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(epi_done);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 bg = b2s[32 + c4 + j], ng = nws[32 + c4 + j];
            apart(gated_value(two(y[4 * j], y[4 * j + 1]), (two(z[4 * j], z[4 * j + 1]) + low(bg)) * (rg2 * low(ng))), y[4 * j], y[4 * j + 1]);
            apart(gated_value(two(y[4 * j + 2], y[4 * j + 3]), (two(z[4 * j + 2], z[4 * j + 3]) + high(bg)) * (rg2 * high(ng))),
                  y[4 * j + 2], y[4 * j + 3]);
          }
          finish(y, 64 * grp + 32 * j2, row0);
        }
      } else {
        // ---------------------------------------------- result of the second contraction (GATED: this group's 64 columns)
        if constexpr (MODE == MLP_GATED_BWD) wait(d2_full, par);
        else wait(d2_full + 8 * grp, par);
        constexpr int NC = GATED ? 2 : 4;
#pragma unroll 1
        for (int c = 0; c < NC; ++c) {
          const int col = GATED ? 64 * grp + 32 * c : 32 * c;
          float y[32];
          tmem_get(lane_q + 128u * reg_d + (uint32_t)col, y);
          if (c == NC - 1) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(epi_done + (GATED ? 0 : 8 * grp));
          }
          if constexpr (FWD) {
            const float4* const b2s = reinterpret_cast<const float4*>(cst + 256) + col / 4;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 v = b2s[j];
              add4_to(y + 4 * j, v);
            }
          }
          finish(y, col, row0);
        }
      }
    }
    if (EPI_RES && !alive) drain_copies(my_full, 2, asked);  // (otherwise it has used all that it asked for)
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    // ---------------------------------------------------------------- producers
    // Warp pw: lane quarter (warp & 3), K chunks of its parity; then the side patches of epilogue warp pw (same quarter).
    pdl_sync();
    const int pw = warp - ML_PROD_WARP0, parity = pw >> 2, quarter = warp & 3;
    const int lr = lane >> 3, lc = lane & 7;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t patch = sm0 + ML_CONV_OFF + pw * ML_PATCH, side0 = sm0 + ML_SIDE_OFF + pw * 2 * ML_PATCH;
    const uint32_t put_even = lr * 128 + ((lc ^ lr) << 4), put_odd = lr * 128 + ((lc ^ (lr | 4)) << 4);
    const int n_seg = d.n_src + (MODE == MLP_GATED_BWD ? d.n_ext : 0);
    bool alive = true;
    uint32_t g = (uint32_t)parity, side_n = 0, conv_n = 0;  // number of this warp's next chunk, side patch, chunk by TMA
    uint32_t conv_asked = 0, side_asked = 0;                // copies asked for: numbers below these
    const uint32_t my_conv = conv_full + 8 * pw;
    auto put = [&](uint32_t p, int i, const float4& v) {  // row lr + 4 i of a patch
      sts4(p + ((i & 1) ? put_odd : put_even) + 512u * i, v.x, v.y, v.z, v.w);
    };
    auto tile_row = [&](int t) { return (first_rt + t * step_rt) * 128 + quarter * 32; };
    auto is_direct = [&](int s) { return (s < d.n_src ? d.src[s].idx : d.ext[s - d.n_src].idx) == nullptr; };
    auto request = [&](int t, int s, int k, bool stored) {  // rows read in place: this warp's chunk k of segment s
      if (!alive) return;
      ++conv_asked;
      if (lane == 0) {
        if (stored) to_async_proxy();  // the patch held gathered rows
        load_patch(s < d.n_src ? &maps.src[s] : &maps.ext[s - d.n_src], patch, my_conv, 32 * (parity + 2 * k), tile_row(t));
      }
    };
    auto wait_empty = [&]() {  // the next side patch may be filled
      if (side_n >= 2 && alive) alive = mbar_wait(side_empty + 8 * (2 * pw + (side_n & 1)), ((side_n >> 1) - 1) & 1);
      alive = __all_sync(0xffffffffu, alive);
    };
    auto request_side = [&](const CUtensorMap* map, int x, int y) {  // the next side patch by TMA
      wait_empty();
      if (alive) {
        side_asked = side_n + 1;
        if (lane == 0) load_patch(map, side0 + (side_n & 1) * ML_PATCH, side_full + 8 * (2 * pw + (side_n & 1)), x, y);
      }
      ++side_n;
    };
    auto residual = [&](int t) {
      if (!has_res) return;
      for (int c = 0; c < (GATED ? 2 : 4); ++c) request_side(&maps.res, (GATED ? 64 * parity : 0) + 32 * c, tile_row(t));
    };
    // Addend sums of a tile.  The loads are latency bound (2 k cycles a batch in the running kernel), so as many as fit in the registers
    // are requested together: up to two addends a patch (32 rows), three half a patch at a time.  The row numbers take one register
    // of a lane (= row) for each addend and are shuffled; they are asked for a tile ahead.  573,894 rows, z1 and z2 kept: three addends 0.665 ->
    // 0.576 ms (nothing kept 0.543 -> 0.42), two and a residual 0.534 -> 0.50, no contraction and three addends 0.580 -> 0.484.
    int32_t nx[N_ADD > 0 ? N_ADD : 1];  // row numbers of the next tile
    auto ask_rows = [&](int t) {
      const int64_t at = tile_row(t) + lane, row = at < n_rows ? at : n_rows - 1;
#pragma unroll
      for (int a = 0; a < N_ADD; ++a) nx[a] = d.add[a].idx ? d.add[a].idx[row] : (int32_t)row;
    };
    auto gather = [&](int t, int col0) {
      constexpr int N = N_ADD, ROWS = N == 3 ? 4 : 8;
      int32_t ix[N > 0 ? N : 1];
#pragma unroll
      for (int a = 0; a < N; ++a) ix[a] = nx[a];
      if (t + 1 < n_tiles) ask_rows(t + 1);
#pragma unroll 1
      for (int c = 0; c < 4; ++c, ++side_n) {
        const int col = col0 + 32 * c + lc * 4;
        const float4 b = reinterpret_cast<const float4*>(cst)[col >> 2];
#pragma unroll
        for (int i0 = 0; i0 < 8; i0 += ROWS) {
          float4 v[N > 0 ? N : 1][ROWS];
#pragma unroll
          for (int a = 0; a < N; ++a)
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
              v[a][i] = ld4(d.add[a].ptr + (int64_t)__shfl_sync(0xffffffffu, ix[a], lr + 4 * (i0 + i)) * d.add[a].ld + col);
          if (i0 == 0) wait_empty();
#pragma unroll
          for (int i = 0; i < ROWS; ++i) {
            float4 s = b;
#pragma unroll
            for (int a = 0; a < N; ++a) s = make_float4(s.x + v[a][i].x, s.y + v[a][i].y, s.z + v[a][i].z, s.w + v[a][i].w);
            put(side0 + (side_n & 1) * ML_PATCH, i0 + i, s);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(side_full + 8 * (2 * pw + (side_n & 1)));
      }
    };
    if (n_seg > 0 && is_direct(0)) request(0, 0, 0, false);
    if constexpr (N_ADD > 0) ask_rows(0);
    asm volatile("bar.sync 5, 512;" ::: "memory");  // the constants are there
    for (int t = 0; t < n_tiles; ++t) {
      const int64_t row0 = tile_row(t);
      // rows past the end repeat the last row; their results are never written
      auto row_of = [&](int i) { const int64_t r = row0 + lr + 4 * i; return r < n_rows ? r : n_rows - 1; };
      // ------------------------------------------------ A operand
      for (int s = 0; s < n_seg; ++s) {
        const mb_src& sr = s < d.n_src ? d.src[s] : d.ext[s - d.n_src];
        const int32_t* const idx = sr.idx;
        const bool act = sr.act != 0;
#pragma unroll 1
        for (int k = 0; k < 2; ++k, g += 2) {
          if (!idx) {
            if (alive) alive = mbar_wait(my_conv, conv_n & 1);
            alive = __all_sync(0xffffffffu, alive);
            ++conv_n;
          } else {
            const float* const base = sr.ptr + sr.col + lc * 4 + 32 * (parity + 2 * k);
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = ld4(base + (int64_t)idx[row_of(i)] * sr.ld);
#pragma unroll
            for (int i = 0; i < 8; ++i) put(patch, i, v[i]);
            __syncwarp();
          }
          float x[32];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 v = lds4(patch + lane * 128 + ((j ^ (lane & 7)) << 4));
            x[4 * j] = v.x; x[4 * j + 1] = v.y; x[4 * j + 2] = v.z; x[4 * j + 3] = v.w;
          }
          if (act) {
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = silu_fast_f(x[i]);
          }
          uint32_t hi[2][8], lo[2][8];
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            float sx[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) sx[i] = x[16 * hh + i];
            split_bf16(sx, hi[hh], lo[hh]);
          }
          const uint32_t ab = g & 3, ta = lane_base + ML_A_BASE + 32u * ab;
          if (g >= 4 && alive) alive = mbar_wait(a_done + 8 * ab, ((g >> 2) - 1) & 1);  // A buffer ab is free again
          alive = __all_sync(0xffffffffu, alive);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            MB_TMEM_ST8(ta + 8 * hh, hi[hh]);
            MB_TMEM_ST8(ta + 16 + 8 * hh, lo[hh]);
          }
          // Every lane has used the values it read from the patch (the stores above depend on them): only now may the copy of the
          // next chunk overwrite it.  Issued right after the reads it could overtake them.
          __syncwarp();
          const int s2 = k == 0 ? s : (s + 1 < n_seg ? s + 1 : 0), t2 = k == 1 && s + 1 == n_seg ? t + 1 : t;
          if (t2 < n_tiles && is_direct(s2)) request(t2, s2, k ^ 1, idx != nullptr);
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(a_ready + 8 * ab);
        }
      }
      // ------------------------------------------------ side patches of epilogue warp pw: four for mid, then the residual's.
      // PLAIN: the residual patches of a tile are consumed after L2(t), which is issued after L1(t + 1), which needs this
      // warp's chunks of tile t + 1: they are requested one tile late.
      if (!GATED && (t & 1) != parity) {
        if (t > 0) residual(t - 1);
        continue;
      }
      const int col0 = GATED ? 128 * parity : 0;
      if constexpr (N_ADD > 0) {
        gather(t, col0);
      } else if constexpr (!FWD) {
        for (int c = 0; c < 4; ++c) request_side(&maps.side, col0 + 32 * c, (int)row0);
      }
      if (MODE == MLP_GATED_BWD) residual(t);
    }
    if (!GATED && ((n_tiles - 1) & 1) == parity) residual(n_tiles - 1);
    if (!alive) drain_copies(my_conv, 1, conv_asked);  // (otherwise it has used all that it asked for)
    drain_copies(side_full + 16 * pw, 2, side_asked);
  }

  // ------------------------------------------------------------------ common exit: release tensor memory
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == ML_MMA_WARP) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(PS_TMEM_COLS) : "memory");
  }
}
