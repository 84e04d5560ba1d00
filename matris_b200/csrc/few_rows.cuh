// Dense layers and two-layer MLPs of few rows (included by gemm.cu inside namespace mb, after linear_tma.cuh).
//
// What bounds a small call is the chain of one tile, not a rate: k_mlp and k_linear walk 128-row tiles through seven or eight
// hand-overs between warp roles, a thread works through a whole row, and all but a few multiprocessors idle (back to back, one tile
// of the gated forward 17.7 us, of its backward 13, a dense layer 6 - 11; here 7.2, 6.5 and 3.3 - 6.2; an evaluation of 4 atoms
// 5.1 -> 3.4 ms).  Here a block takes R = 16, 32 or 64 rows and the product is TRANSPOSED, features x
// rows:
//
//   D^T [128 features, R rows] = W [128, K] x X^T       M = 128 weight rows (A, by TMA), N = rows (B, K-major, converted by threads)
//
// so that the matrix instruction's M is always full, however few the rows, and its time shrinks with them.  With thread = feature
// (tensor-memory lane) and registers = rows, bias and weights of an epilogue are one register, a row of an addend table, gate,
// residual or output is one 128-byte access of a warp straight from or to global memory (no staging, no hand-over), and the hidden
// layer goes back to shared memory as the MN-major B operand of layer 2.  A feature's rows are spread over 16 warps.  A table's row
// numbers are asked for first of all, in one register of a lane each, and shuffled: three addends without a contraction 6.2 -> 5.8 us for
// 16 rows, 13.2 -> 12.6 for 9,472; with K = 128 7.0 -> 7.1 and 15.6 -> 14.8.
//
// The products of a K step are accumulated in the order of the persistent kernels, so that a row's sums do not depend on how many rows
// a call has.  (w_hi x [x_hi ; x_lo] as one instruction of N = 2 R, the small terms in columns of their own, would save a third of the
// matrix instructions' time, but rounds differently.)
//
// One tile per block and every barrier used once, but for the ring of weight slots (32 KB: hi and lo of 64 K values).  Inside an
// evaluation the weights are asked for before the wait for the preceding kernel (`early`, see common.cuh): by the time its
// results are there, up to 128 KB of them are on chip.
//
// Warps 0 - 15: rows in, epilogues; 16: matrix instructions; 17: weights.

// A small evaluation is also bound by its launches, 2.5 us of the host's time each and 3 - 4 of the chain, so a launch takes on
// more: ROW_BWD is the backward pass from a row's own gradient on (RowBwd, common.cuh), a warp forming the row's dz2 (and the
// logits' gradients) in registers as the row kernels do; LINEAR takes the column blocks of independent problems, and sums of a
// bond's two directed rows as operand; PLAIN_BWD two problems.  With the envelopes' (evaluate.cu) an evaluation of 4 atoms takes 443
// launches instead of 660 (32 atoms 494, 572 atoms 599), 3.37 -> 2.91 ms, of 32 atoms through the calculator 5.02 -> 4.84.  Left out
// again one by one: row gradients 3.0 and 0.4 % slower, LINEAR's problems 5.2 and 2.6 %, PLAIN_BWD's 2.7 and 1.2 %; 572 atoms, where
// few launches are of few rows, within 0.3 %.

enum FewMode { FEW_GATED_FWD = MLP_GATED_FWD, FEW_PLAIN_FWD = MLP_PLAIN_FWD, FEW_GATED_BWD = MLP_GATED_BWD,
               FEW_PLAIN_BWD = MLP_PLAIN_BWD, FEW_LINEAR = 4, FEW_ROW_BWD = 5 };
constexpr int FW_MAX_BLOCKS = 8;
struct FewLinear { mb_colblock blk[FW_MAX_BLOCKS]; int64_t n_rows[FW_MAX_BLOCKS]; const int32_t* pair; };  // independent problems' column blocks
struct FewPlainBwd { MlpArgs of[2]; };                                                                     // two independent problems
struct FewRowBwd : MlpArgs { RowGrad g; float* out[3]; float* zero; int64_t n_zero; };
template <int MODE> struct FewArgs { typedef MlpArgs T; };
template <> struct FewArgs<FEW_LINEAR> { typedef FewLinear T; };
template <> struct FewArgs<FEW_PLAIN_BWD> { typedef FewPlainBwd T; };
template <> struct FewArgs<FEW_ROW_BWD> { typedef FewRowBwd T; };
template <typename T> __device__ __forceinline__ const T& few_problem(const T& args, int) { return args; }  // that of a block
__device__ __forceinline__ const MlpArgs& few_problem(const FewPlainBwd& args, int i) { return args.of[i]; }
// hi, lo; MLPs: layer 1, layer 2, E's weights (PLAIN_BWD: two of each problem); LINEAR: column blocks
struct alignas(64) FewMaps { CUtensorMap w[FW_MAX_BLOCKS][2]; };

constexpr int FW_WORKERS = 16, FW_MMA_WARP = 16, FW_TMA_WARP = 17, FW_THREADS = 576;
constexpr uint32_t FW_SMEM_LIMIT = 227 * 1024;
constexpr uint32_t FW_SLOT_BYTES = 2 * TC_TILE_BYTES, FW_MAX_SLOTS = 6;
// Operands are 128-byte cores (8 rows x 8 K, or 8 K x 8 rows) in the order of K; bytes of 8 rows x 128 K of an operand part:
constexpr uint32_t FW_GROUP = 2048;
constexpr uint32_t FW_ROW_CORE = 144, FW_ROW_GROUP = 16 * FW_ROW_CORE;  // ROW_BWD, whose warps write along K: 16 bytes between cores

// shared memory: weight ring | X segments | hidden layer | sums of squares | barriers.  A branch's hidden layer takes the place of an X
// segment whose products are done by then (GATED_FWD: the gate's, whose segments serve the core as well).
__host__ __device__ constexpr uint32_t few_operand_bytes(int r) { return (uint32_t)r * 512u; }  // hi and lo of R rows x 128 K
__host__ __device__ constexpr uint32_t few_x_bytes(int mode, int r) { return (uint32_t)(r / 4) * (mode == FEW_ROW_BWD ? FW_ROW_GROUP : FW_GROUP); }
__host__ __device__ constexpr int few_hidden(int mode, int n_src) { return mode != FEW_GATED_FWD ? 0 : n_src > 0 ? 1 : 2; }  // of its own
__host__ __device__ constexpr uint32_t few_tail_bytes(int r) { return (uint32_t)r * 32u + 256u; }
__host__ __device__ constexpr uint32_t few_columns(int mode, int r) {
  const uint32_t need = (uint32_t)r * (mode == FEW_GATED_FWD ? 4 : mode == FEW_GATED_BWD || mode == FEW_ROW_BWD ? 3 : mode == FEW_LINEAR ? 1 : 2);
  return need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512;
}

// no swizzle: LBO = bytes between cores along K, SBO = between groups of 8 rows (both majors)
__device__ __forceinline__ uint64_t few_desc(uint32_t saddr, uint32_t core = 128, uint32_t group = FW_GROUP) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)(core >> 4) << 16 | (uint64_t)(group >> 4) << 32 | 1ull << 46;
}
// four consecutive K values of a row (c8: their core, second half of it or not) into an operand's hi and lo part
__device__ __forceinline__ void few_put4(uint32_t at, uint32_t lo_off, const float4& v) {
  const float x[4] = {v.x, v.y, v.z, v.w};
  uint32_t hi[2], lo[2];
  split_bf16(x, hi, lo);
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" :: "r"(at), "r"(hi[0]), "r"(hi[1]) : "memory");
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" :: "r"(at + lo_off), "r"(lo[0]), "r"(lo[1]) : "memory");
}
__device__ __forceinline__ void umma_bf16_ss(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               :: "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
template <int N> __device__ __forceinline__ void few_tmem_ld(uint32_t addr, uint32_t (&v)[N]) {
  static_assert(N == 4 || N == 8, "rows of a thread");
  if constexpr (N == 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr) : "memory");
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
template <int RT> __device__ __forceinline__ void few_result(uint32_t addr, float (&y)[RT]) {
  uint32_t a[RT];
  few_tmem_ld(addr, a);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < RT; ++i) y[i] = __uint_as_float(a[i]);
}
// V sums of squares over the 32 lanes at once: lane l ends with that of value l / (32 / V) (V - 1 + log2(32 / V) shuffles).  The order
// of the additions is that of sum_of_squares() in mlp_fused.cuh.
template <int V> __device__ __forceinline__ float few_sums_of_squares(float (&v)[V], int lane) {
  int o = 16;
#pragma unroll
  for (int n = V / 2; n > 0; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float own = up ? v[i + n] : v[i], other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + n], o);
      if (2 * n == V) {
        const float lower = up ? other : own, upper = up ? own : other;
        v[i] = fmaf(upper, upper, __fmul_rn(lower, lower));
      } else {
        v[i] = own + other;
      }
    }
  }
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

template <int MODE, int R>
__global__ void __launch_bounds__(FW_THREADS, MODE == FEW_LINEAR ? 2 : 1)
k_few(const __grid_constant__ typename FewArgs<MODE>::T args, const __grid_constant__ FewMaps maps, const int n_slots, const int early) {
  constexpr bool LINEAR = MODE == FEW_LINEAR, ROW_BWD = MODE == FEW_ROW_BWD;
  constexpr bool GATED_BWD = MODE == FEW_GATED_BWD || ROW_BWD, GATED = MODE == FEW_GATED_FWD || GATED_BWD;
  constexpr bool FWD = MODE == FEW_GATED_FWD || MODE == FEW_PLAIN_FWD;
  constexpr int NB = GATED ? 2 : 1, RT = R < 32 ? R / 4 : 8, NCH = R < 32 ? 1 : R / 32;  // rows of a thread: NCH times RT
  constexpr int JOBS = R / 2;                                                           // (8 rows x 32 values) pieces of a segment
  constexpr uint32_t OPERAND = few_operand_bytes(R), LO = (R / 8) * FW_GROUP;  // of the hidden layer
  constexpr uint32_t X_CORE = ROW_BWD ? FW_ROW_CORE : 128, X_GROUP = ROW_BWD ? FW_ROW_GROUP : FW_GROUP;
  constexpr uint32_t X_OPERAND = few_x_bytes(MODE, R), X_LO = X_OPERAND / 2;
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)R >> 3) << 17 | ((128u >> 4) << 24), MN_MAJOR_B = 1u << 16;
  constexpr uint32_t COLUMNS = few_columns(MODE, R);
  const auto& d = few_problem(args, blockIdx.y);
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sm0 = smem_u32(smem);
  if ((sm0 & 1023u) != 0) {
    if (threadIdx.x == 0) atomicOr(&g_gemm_status, 2);
    return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int64_t n_rows;
  if constexpr (LINEAR) n_rows = d.n_rows[blockIdx.y];
  else n_rows = d.n_rows;
  const int64_t row0 = (int64_t)blockIdx.x * R;
  if (row0 >= n_rows) return;  // (another problem of the launch has more rows)
  int n_src, n_ext = 0;  // segments of layer 1 (GATED_BWD: core and gate half of dz2); of E
  if constexpr (LINEAR) n_src = d.blk[blockIdx.y].n_src;
  else n_src = d.n_src;
  if constexpr (GATED_BWD) n_ext = d.n_ext;
  bool two_layers = !LINEAR;
  if constexpr (ROW_BWD) two_layers = d.out[0] != nullptr;
  const int n_seg = n_src + n_ext;

  const uint32_t x_sm = sm0 + n_slots * FW_SLOT_BYTES, own_sm = x_sm + n_seg * X_OPERAND, ss_off = own_sm + few_hidden(MODE, n_src) * OPERAND - sm0;
  auto hidden_at = [&](uint32_t x, uint32_t own, int br) {  // a branch's hidden layer
    if constexpr (MODE == FEW_GATED_FWD) return br == 0 ? own : n_src > 0 ? x : own + OPERAND;
    else return x + br * X_OPERAND;
  };
  float* const sums = reinterpret_cast<float*>(smem + ss_off);  // [8 rows x 4][row quarter][value][lane quarter]
  const uint32_t bar0 = sm0 + ss_off + R * 32;
  // w_full[6] w_empty[6] | x_ready[4] (per segment) | act_ready[2] d1_full[2] d2_full[2] | retired | tensor-memory address
  const uint32_t w_full = bar0, w_empty = bar0 + 48, x_ready = bar0 + 96, act_ready = bar0 + 128, d1_full = bar0 + 144,
                 d2_full = bar0 + 160, retired = bar0 + 176, slot_at = bar0 + 184;
  if (warp == FW_MMA_WARP) {
    if (lane == 0) {
      for (uint32_t b = 0; b < FW_MAX_SLOTS; ++b) { mbar_init(w_full + 8 * b, 1); mbar_init(w_empty + 8 * b, 1); }
      for (int b = 0; b < 4; ++b) mbar_init(x_ready + 8 * b, ROW_BWD ? FW_WORKERS : JOBS);
      for (int b = 0; b < 2; ++b) { mbar_init(act_ready + 8 * b, FW_WORKERS); mbar_init(d1_full + 8 * b, 1); mbar_init(d2_full + 8 * b, 1); }
      mbar_init(retired, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(slot_at), "r"(COLUMNS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  uint32_t tmem_base;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(slot_at) : "memory");

  // The sequence of 64-value K pieces of weights: step(number, layer, branch, piece).  Layer 2 stands for E.
  auto walk = [&](auto step) {
    int n = 0;
    for (int br = 0; br < NB; ++br)
      for (int kp = 0; kp < (GATED_BWD ? 2 : 2 * n_src); ++kp) step(n++, 0, br, kp);
    for (int kp = 0; kp < 2 * n_ext; ++kp) step(n++, 2, 0, kp);
    if (two_layers)
      for (int br = 0; br < NB; ++br)
        for (int kp = 0; kp < 2; ++kp) step(n++, 1, br, kp);
  };

  if (warp == FW_MMA_WARP) {
    // The chain's longest part: 12 instructions a piece of 64 K values, 40 cycles each for N <= 32 (A is read from shared memory), if
    // the loop around them stays short (slots counted up, no division, descriptors stepped): 1100 -> 720 cycles a piece.
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0), sm_u = __shfl_sync(0xffffffffu, sm0, 0);
    const uint32_t x_u = sm_u + n_slots * FW_SLOT_BYTES, own_u = x_u + n_seg * X_OPERAND;
    const uint64_t w_first = umma_desc(sm_u);
    bool alive = true;
    uint32_t slot = 0, phase = 0;  // of the next piece
    auto wait = [&](uint32_t bar, uint32_t parity) { if (alive) alive = mbar_wait(bar, parity); };
    // one piece: rows' descriptors (hi; lo is `lo` further on), step of 16 K values
    auto piece = [&](uint32_t dt, uint64_t xh, uint32_t lo, uint32_t adv, uint32_t idesc, bool fresh) {
      wait(w_full + 8 * slot, phase);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elected) {
        const uint64_t wh = w_first + slot * (FW_SLOT_BYTES >> 4), wl = wh + (TC_TILE_BYTES >> 4), xl = xh + (lo >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {  // K steps of 16: 32 bytes of the weight rows, two cores of the rows
          umma_bf16_ss(dt, wh + 2 * kk, xl + adv * kk, idesc, (!fresh || kk > 0) ? 1u : 0u);
          umma_bf16_ss(dt, wl + 2 * kk, xh + adv * kk, idesc, 1u);
          umma_bf16_ss(dt, wh + 2 * kk, xh + adv * kk, idesc, 1u);
        }
        mma_commit(w_empty + 8 * slot);
      }
      __syncwarp();
      if (++slot == (uint32_t)n_slots) { slot = 0; phase ^= 1; }
    };
    auto segment = [&](int seg, uint32_t dt, bool fresh) {  // both pieces of an X segment
      wait(x_ready + 8 * seg, 0);
      const uint64_t xh = few_desc(x_u + seg * X_OPERAND, X_CORE, X_GROUP);
#pragma unroll 1
      for (int kp = 0; kp < 2; ++kp) piece(dt, xh + kp * (8 * X_CORE / 16), X_LO, 2 * X_CORE / 16, IDESC, fresh && kp == 0);
    };
    auto full = [&](uint32_t bar) {
      if (elected) mma_commit(bar);
      __syncwarp();
    };
#pragma unroll 1
    for (int br = 0; br < NB; ++br) {
#pragma unroll 1
      for (int s = 0; s < (GATED_BWD ? 1 : n_src); ++s) segment(GATED_BWD ? br : s, tmem_u + R * br, s == 0);
      if (n_src > 0) full(LINEAR ? d2_full : d1_full + 8 * br);
    }
#pragma unroll 1
    for (int s = 0; s < n_ext; ++s) segment(n_src + s, tmem_u + 2 * R, s == 0);
    if (two_layers) {
#pragma unroll 1
      for (int br = 0; br < NB; ++br) {
        wait(act_ready + 8 * br, 0);
        const uint32_t dt = tmem_u + R * (MODE == FEW_GATED_FWD ? 2 + br : NB);
        const uint64_t ah = few_desc(hidden_at(x_u, own_u, br));
#pragma unroll 1
        for (int kp = 0; kp < 2; ++kp)
          piece(dt, ah + kp * (1024 / 16), LO, 16, IDESC | MN_MAJOR_B, kp == 0 && !(GATED_BWD && (br == 1 || n_ext > 0)));
        if (!GATED_BWD || br == 1) full(d2_full + (MODE == FEW_GATED_FWD ? 8 * br : 0));
      }
    }
    drain_mma(retired, elected);
  } else if (warp == FW_TMA_WARP) {
    if (!early) pdl_sync();
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    const uint32_t sm_u = __shfl_sync(0xffffffffu, sm0, 0);
    bool alive = true;
    uint32_t asked = 0;
    walk([&](int n, int layer, int br, int kp) {
      const int slot = n % n_slots;
      if (n >= n_slots && alive) alive = mbar_wait(w_empty + 8 * slot, (uint32_t)(n / n_slots - 1) & 1);
      alive = __all_sync(0xffffffffu, alive);
      if (!alive) return;
      // the rows of a branch's weights, but W1t of the gated backward has its branches side by side (and 128 rows for every output)
      const bool beside = GATED_BWD && layer == 1;
      const int x = 64 * kp + (beside ? 128 * br : 0), y = beside ? 128 * (int)blockIdx.y : 128 * br;
      if (elected) {
        const CUtensorMap* const m = maps.w[LINEAR ? (int)blockIdx.y : MODE == FEW_PLAIN_BWD ? 2 * (int)blockIdx.y + layer : layer];
        const uint32_t bar = w_full + 8 * slot, dst = sm_u + slot * FW_SLOT_BYTES;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(FW_SLOT_BYTES) : "memory");
        tma_load_2d(dst, m, bar, x, y);
        tma_load_2d(dst + TC_TILE_BYTES, m + 1, bar, x, y);
      }
      __syncwarp();
      ++asked;
    });
    drain_copies(w_full, (uint32_t)n_slots, asked);
  } else {
    // ---------------------------------------------------------------- workers
    const int q = warp & 3, rg = warp >> 2, f = 32 * q + lane, r0 = rg * RT;  // first row of chunk 0; chunk c: 32 c further on
    const uint32_t lane_q = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)r0;
    bool alive = true;
    auto wait = [&](uint32_t bar) {
      if (alive) alive = mbar_wait(bar, 0);
      alive = __all_sync(0xffffffffu, alive);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    auto row_of = [&](int c, int i) { const int64_t r = row0 + 32 * c + r0 + i; return r < n_rows ? r : n_rows - 1; };  // (past the end: the last)
    auto store = [&](float* p, int64_t ld, int c, const float (&v)[RT]) {
      const int64_t first = row0 + 32 * c + r0, n = alive ? n_rows - first : 0;
#pragma unroll
      for (int i = 0; i < RT; ++i)
        if (i < n) p[(first + i) * ld] = v[i];
    };
    pdl_sync();
    float side[NCH][NB][RT], res[RT];  // what the epilogues add or multiply with; the residual's rows of a chunk
    bool has_res = false;
    if constexpr (!LINEAR) has_res = ROW_BWD ? d.res != nullptr && blockIdx.y == 0 : d.out2 != nullptr;
    auto ask_res = [&](int c) {
      if constexpr (!LINEAR) {
#pragma unroll
        for (int i = 0; i < RT; ++i) res[i] = d.res[row_of(c, i) * d.ld_res + f];
      }
    };
    auto ask_side = [&]() {
      if constexpr (!LINEAR && !FWD) {
#pragma unroll
        for (int c = 0; c < NCH; ++c)
#pragma unroll
          for (int br = 0; br < NB; ++br)
#pragma unroll
            for (int i = 0; i < RT; ++i) side[c][br][i] = d.side[row_of(c, i) * d.ld_side + 128 * br + f];
      }
      if constexpr (!LINEAR) {
        if (has_res && NCH == 1) ask_res(0);
      }
    };
    int32_t ix[3] = {0, 0, 0};  // row numbers of the addends: lane RT c + i has row i of chunk c
    if constexpr (MODE == FEW_GATED_FWD) {
      const int64_t at = row0 + 32 * (lane / RT) + r0 + lane % RT, r = at < n_rows ? at : n_rows - 1;
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (a < d.n_add) ix[a] = d.add[a].idx ? d.add[a].idx[r] : (int32_t)r;
    }
    if constexpr (ROW_BWD) {
      // -------------------------------------------- X: a row per warp and turn, lane = 4 channels
      ask_side();
#pragma unroll
      for (int n0 = 0; n0 < R; n0 += FW_WORKERS) {
        const int n = n0 + warp, c = 4 * lane;
        const bool mine = row0 + n < n_rows;
        const int64_t row = mine ? row0 + n : n_rows - 1;
        const uint32_t at = x_sm + (n >> 3) * FW_ROW_GROUP + (lane >> 1) * FW_ROW_CORE + (n & 7) * 16u + (lane & 1) * 8u;
        float4 o, ds, dt;
        if (d.g.kind == 1) {
          attn_bwd_row(d.g, row, c, o, ds, dt);
          if (n_ext > 0) {
            few_put4(at + 2 * X_OPERAND, X_LO, ds);
            few_put4(at + 3 * X_OPERAND, X_LO, dt);
          }
          if (d.g.dlogits && mine) {
            st4(d.g.dlogits + row * 256 + c, ds);
            st4(d.g.dlogits + row * 256 + 128 + c, dt);
          }
        } else if (d.g.kind == 2) {
          o = smooth_bwd_row(d.g, row, c);
        } else {
          o = ld4(d.g.dh_in + row * 128 + c);
        }
        gate_bwd_row(d.g.z2 + row * 256, c, d.g.norm_core, d.g.norm_gate, o, ds, dt);
        few_put4(at, X_LO, ds);
        few_put4(at + X_OPERAND, X_LO, dt);
      }
      to_async_proxy();
      __syncwarp();
      if (lane < n_seg) mbar_arrive(x_ready + 8 * lane);
      if (blockIdx.y == 0)
        for (int64_t i = 4 * ((int64_t)blockIdx.x * (32 * FW_WORKERS) + tid); i < d.n_zero; i += 4 * (int64_t)gridDim.x * (32 * FW_WORKERS))
          st4(d.zero + i, make_float4(0.f, 0.f, 0.f, 0.f));
    } else
    // ---------------------------------------------- X: 8 rows x 32 values per warp and turn, lane = (row, 8 values)
    for (int j = warp; j < n_seg * JOBS; j += FW_WORKERS) {
      const int seg = j / JOBS, piece = j % JOBS, n = 8 * (piece >> 2) + (lane & 7), c8 = 4 * (piece & 3) + (lane >> 3);
      const mb_src* sr;
      if constexpr (LINEAR) sr = &d.blk[blockIdx.y].src[seg];
      else sr = seg < n_src ? &d.src[seg] : &d.ext[seg - n_src];
      int64_t r = row0 + n < n_rows ? row0 + n : n_rows - 1;
      if (sr->idx) r = sr->idx[r];
      const float* const p = sr->ptr + r * sr->ld + sr->col + 8 * c8;
      float4 u = ld4(p), v = ld4(p + 4);
      if constexpr (LINEAR) {
        if (d.pair) {
          const float* const p2 = sr->ptr + (int64_t)d.pair[r] * sr->ld + sr->col + 8 * c8;
          u = add4(u, ld4(p2));
          v = add4(v, ld4(p2 + 4));
        }
      }
      float x[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
      if (sr->act) {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = silu_fast_f(x[i]);
      }
      uint32_t hi[4], lo[4];
      split_bf16(x, hi, lo);
      const uint32_t at = x_sm + seg * OPERAND + (n >> 3) * FW_GROUP + c8 * 128u + (n & 7) * 16u;
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(at), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(at + LO), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
      to_async_proxy();
      __syncwarp();
      if (lane == 0) mbar_arrive(x_ready + 8 * seg);
    }
    if constexpr (LINEAR) {
      const mb_colblock& cb = d.blk[blockIdx.y];
      const float bias = cb.bias ? cb.bias[f] : 0.f, rw = cb.res && cb.res_w ? cb.res_w[f] : 1.f, sc = cb.out_scale;
      float* const out = cb.out + cb.col_out + f;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        float g[RT], x[RT], y[RT];
        if (cb.gate) {
#pragma unroll
          for (int i = 0; i < RT; ++i) g[i] = cb.gate[row_of(c, i) * cb.ld_gate + cb.col_gate + f];
        }
        if (cb.res) {
#pragma unroll
          for (int i = 0; i < RT; ++i) x[i] = cb.res[row_of(c, i) * cb.ld_res + cb.col_res + f];
        }
        if (c == 0) wait(d2_full);
        few_result(lane_q + 32u * c, y);
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          y[i] += bias;
          if (cb.gate) y[i] *= silu_grad_fast_f(g[i]);
          if (cb.out_act) y[i] = silu_fast_f(y[i]);
          if (cb.res) y[i] = fmaf(rw, x[i], y[i]);
          y[i] *= sc;
        }
        if (cb.mode == MB_OUT_STORE) {
          store(out, cb.ld_out, c, y);
        } else {  // one addition per element at the memory side; every row has one writer
          const int64_t first = row0 + 32 * c + r0, n = alive ? n_rows - first : 0;
#pragma unroll
          for (int i = 0; i < RT; ++i)
            if (i < n) atomicAdd(out + (first + i) * cb.ld_out, y[i]);
        }
      }
    } else {
      // -------------------------------------------- what the epilogues add, on its way while the first products are formed
      if constexpr (FWD) {
#pragma unroll
        for (int br = 0; br < NB; ++br) {
          const float b = d.b1 ? d.b1[128 * br + f] : 0.f;
#pragma unroll
          for (int c = 0; c < NCH; ++c)
#pragma unroll
            for (int i = 0; i < RT; ++i) side[c][br][i] = b;
        }
        if constexpr (GATED) {
#pragma unroll
          for (int a = 0; a < 3; ++a)
            if (a < d.n_add) {
              const mb_add& t = d.add[a];
              float v[NCH][NB][RT];
#pragma unroll
              for (int c = 0; c < NCH; ++c)
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                  const float* const p = t.ptr + (int64_t)__shfl_sync(0xffffffffu, ix[a], RT * c + i) * t.ld + f;
#pragma unroll
                  for (int br = 0; br < NB; ++br) v[c][br][i] = p[128 * br];
                }
#pragma unroll
              for (int c = 0; c < NCH; ++c)
#pragma unroll
                for (int br = 0; br < NB; ++br)
#pragma unroll
                  for (int i = 0; i < RT; ++i) side[c][br][i] += v[c][br][i];
            }
        }
      }
      if constexpr (!ROW_BWD) ask_side();
      // -------------------------------------------- layer 1 out, hidden layer back as the operand of layer 2
#pragma unroll
      for (int br = 0; br < NB; ++br) {
        float x[NCH][RT];
        if (!FWD || n_src > 0) wait(d1_full + 8 * br);
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          if (!FWD || n_src > 0) {
            few_result(lane_q + (uint32_t)R * br + 32u * c, x[c]);
          } else {
#pragma unroll
            for (int i = 0; i < RT; ++i) x[c][i] = 0.f;
          }
          float a[RT];
#pragma unroll
          for (int i = 0; i < RT; ++i) {
            if constexpr (FWD) {
              x[c][i] += side[c][br][i];
              a[i] = silu_fast_f(x[c][i]);
            } else {
              x[c][i] *= (MODE == FEW_PLAIN_BWD ? d.scale : 1.f) * silu_grad_fast_f(side[c][br][i]);
              a[i] = x[c][i];
            }
          }
          if (!two_layers) continue;
          uint32_t hi[RT / 2], lo[RT / 2];
          split_bf16(a, hi, lo);
          const int n = 32 * c + r0;
          const uint32_t at = hidden_at(x_sm, own_sm, br) + (n >> 3) * FW_GROUP + f * 16u + (n & 7) * 2u;
          if constexpr (RT == 8) {
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(at), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" :: "r"(at + LO), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
          } else {
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" :: "r"(at), "r"(hi[0]), "r"(hi[1]) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" :: "r"(at + LO), "r"(lo[0]), "r"(lo[1]) : "memory");
          }
        }
        if (two_layers) {
          to_async_proxy();
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(act_ready + 8 * br);
        }
        if (d.z1) {
#pragma unroll
          for (int c = 0; c < NCH; ++c) store(d.z1 + 128 * br + f, d.ld_z1, c, x[c]);
        }
      }
      // -------------------------------------------- layer 2 out
      if (two_layers) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          float y[RT];
          if (has_res && NCH > 1) ask_res(c);
          if constexpr (MODE == FEW_GATED_FWD) {
            float z[2][RT], v[2 * RT];
#pragma unroll
            for (int br = 0; br < 2; ++br) {
              const float b = d.b2 ? d.b2[128 * br + f] : 0.f;
              if (c == 0) wait(d2_full + 8 * br);
              few_result(lane_q + (uint32_t)R * (2 + br) + 32u * c, z[br]);
#pragma unroll
              for (int i = 0; i < RT; ++i) {
                z[br][i] += b;
                v[RT * br + i] = z[br][i];
              }
              if (d.z2) store(d.z2 + 128 * br + f, d.ld_z2, c, z[br]);
            }
            constexpr int PER = 32 / (2 * RT);  // lanes that end with the same sum
            const float s = few_sums_of_squares(v, lane);
            float* const mine = sums + (c * 4 + rg) * 8 * RT;
            if (lane % PER == 0) mine[(lane / PER) * 4 + q] = s;
            asm volatile("bar.sync %0, 128;" :: "r"(1 + rg) : "memory");  // the four lane quarters of these rows
            const float nc = d.norm_core[f], ng = d.norm_gate[f];
#pragma unroll
            for (int i = 0; i < RT; ++i) {
              const float4 sc = *reinterpret_cast<const float4*>(mine + 4 * i);
              const float4 sg = *reinterpret_cast<const float4*>(mine + 4 * (RT + i));
              const float rc = rsqrtf(((sc.x + sc.y) + (sc.z + sc.w)) * (1.0f / 128.0f) + ML_RMS_EPS);
              const float rr = rsqrtf(((sg.x + sg.y) + (sg.z + sg.w)) * (1.0f / 128.0f) + ML_RMS_EPS);
              y[i] = gated_value(z[0][i] * (rc * nc), z[1][i] * (rr * ng));
            }
          } else {
            const float b = FWD && d.b2 ? d.b2[f] : 0.f;
            if (c == 0) wait(d2_full);
            few_result(lane_q + (uint32_t)R * NB + 32u * c, y);
#pragma unroll
            for (int i = 0; i < RT; ++i) y[i] += b;
          }
          if constexpr (!ROW_BWD) {
            if (d.h) store(d.h + f, d.ld_h, c, y);
          }
          if (has_res) {
            const float rw = d.res_w ? d.res_w[f] : 1.f;
#pragma unroll
            for (int i = 0; i < RT; ++i) y[i] = fmaf(rw, res[i], y[i]);
            if constexpr (!ROW_BWD) store(d.out2 + f, d.ld_out2, c, y);
          }
          if constexpr (ROW_BWD) store(d.out[blockIdx.y] + f, 128, c, y);
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == FW_MMA_WARP) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(COLUMNS) : "memory");
  }
}
