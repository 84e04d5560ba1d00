// Row GEMM with direct outputs (included by gemm.cu inside namespace mb, after mlp_fused.cuh): the descriptors of mb_gemm whose
// column blocks share one A operand or have a single 128-wide segment each and whose outputs go to their own rows (store or
// accumulate, no index).  Those are all dense layers of an evaluation but those of few rows (k_few); scattered outputs take k_gemm_ps.
//
// Same machinery as k_mlp (see there): rows by TMA patches in both directions, A split into bf16 hi / lo in four tensor-memory
// buffers, weights in 16 KB tiles, three accumulator regions used in turn by the column blocks in the order they are finished,
// two groups of four epilogue warps taking alternate blocks.  The gate and residual rows of the epilogue are fetched by a warp of
// their own (18), one lane per epilogue warp, so that they never hold up the A operand of the next tile.
//
// A tile of rows converts its A once for all its column blocks: with K = 128 the blocks run one after another from the resident
// buffers, with a wider K they advance together, chunk pair by chunk pair (at most three, one per region).  Few tiles (the column
// blocks of all of them fit the SMs at once): one CTA per (tile, column block), which shortens the chain where only latency
// counts.
//
// HBM bounds the large launches: 573,894 rows take 0.171 ms for 128 -> 256 (k_gemm_ps 0.214), 0.25 with a gate, 0.36 for
// 512 -> 128, 0.275 for 128 -> 512.  The smallest launches that k_few leaves are bound by the chain of a tile, back to back 6.8 us for 128 -> 128
// (9,473 rows), 11.4 for 512 -> 128 (4,737 rows), whose tile has 16 chunks, 6.9 for 128 -> 512 (2,369 rows).
//
// PAIR sums the two directed rows of a bond on the way in, instead of a pass that writes the sums and one that reads them back: with
// K = 512, 117,048 bonds 98 + 87 -> 115 us (92 at the copy rate), with K = 256 49 + 49 -> 62.  The rows are gathered by cp.async
// into two patches of a producer warp, the next chunk's while this one is converted.  (Through registers 153 and 82 us: beside this
// kernel's shared memory the L1 keeps 28 KB, which is less than the lines the loads of eight warps wait for.)

struct alignas(64) LinMaps {
  CUtensorMap w[4][2];                       // weights of a column block: hi, lo
  CUtensorMap src[4];                        // shared A: segments; otherwise the segment of each block
  CUtensorMap gate[4], res[4], out[4];
};

constexpr int LN_THREADS = 608;              // 19 warps
constexpr int LN_SIDE_WARP = 18;
constexpr int LN_CONST_OFF = ML_STAGE_OFF + 8 * ML_PATCH;   // bias[4][128], res_w[4][128]
constexpr int LN_BAR_OFF = LN_CONST_OFF + 1024 * 4;
constexpr int LN_SMEM_BYTES = LN_BAR_OFF + 640;
static_assert(LN_SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ void copy16(uint32_t to, const float* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(to), "l"(from) : "memory");
}
// PAIR: an operand row is the sum of rows i and pair[i], i = idx[r], one idx for all segments
template <bool PAIR>
__global__ void __launch_bounds__(LN_THREADS, 1)
k_linear(const __grid_constant__ mb_gemm_desc d, const __grid_constant__ LinMaps maps, const int shared_a, const int split,
         const int32_t* const pair) {
  constexpr uint32_t SLOTS = PAIR ? 1 : 2;  // gate / residual patches of an epilogue warp; PAIR: the other one holds its producer's second rows
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + LN_BAR_OFF);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + LN_BAR_OFF + 632);
  const uint32_t sm0 = smem_u32(smem);
  if ((sm0 & 1023u) != 0) {
    if (threadIdx.x == 0) atomicOr(&g_gemm_status, 2);
    return;
  }
  // a_ready[4] (4 producer warps) a_done[4] | w_ready[5] w_done[5] | d_full[6] d_free[6] (4 epilogue warps; block number mod 6:
  // always the same region and the same group) | side_full[8][2] side_empty[8][2] | conv_full[8] | retired
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t a_ready = bar0, a_done = bar0 + 32, w_ready = bar0 + 64, w_done = bar0 + 104, d_full = bar0 + 144,
                 d_free = bar0 + 192, side_full = bar0 + 256, side_empty = bar0 + 384, conv_full = bar0 + 512,
                 retired = bar0 + 576;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* const cst = reinterpret_cast<float*>(smem + LN_CONST_OFF);
  const int64_t n_rows = d.n_rows;
  const int n_row_tiles = (int)((n_rows + 127) >> 7), nb_all = d.n_blocks;
  const int j0 = split ? (int)(blockIdx.x % (unsigned)nb_all) : 0, nb = split ? 1 : nb_all;  // this CTA's column blocks
  const int first_rt = split ? (int)(blockIdx.x / (unsigned)nb_all) : (int)blockIdx.x;
  const int step_rt = split ? n_row_tiles : (int)gridDim.x;  // split: one tile
  const int n_tiles = (n_row_tiles - first_rt + step_rt - 1) / step_rt;
  const int n_kp = 2 * d.blk[0].n_src;                       // chunk pairs per column block
  const int n_seg = shared_a ? d.blk[0].n_src : nb;          // 128-wide A segments per tile
  const int n_kpa = 2 * n_seg;
  auto segment = [&](int s) -> const mb_src& { return shared_a ? d.blk[0].src[s] : d.blk[j0 + s].src[0]; };

  if (warp == ML_MMA_WARP) {
    if (lane == 0) {
      for (int b = 0; b < 4; ++b) { mbar_init(a_ready + 8 * b, 4); mbar_init(a_done + 8 * b, 1); }
      for (uint32_t b = 0; b < ML_W_SLOTS; ++b) { mbar_init(w_ready + 8 * b, 1); mbar_init(w_done + 8 * b, 1); }
      for (int b = 0; b < 6; ++b) { mbar_init(d_full + 8 * b, 1); mbar_init(d_free + 8 * b, 4); }
      for (int b = 0; b < 16; ++b) { mbar_init(side_full + 8 * b, 1); mbar_init(side_empty + 8 * b, 1); }
      for (int b = 0; b < 8; ++b) mbar_init(conv_full + 8 * b, 1);
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

  // step(tile, block, pair): the order both issuing warps walk
  auto walk = [&](auto step) {
    for (int t = 0; t < n_tiles; ++t) {
      if (shared_a && n_kp > 2) {
        for (int kp = 0; kp < n_kp; ++kp)
          for (int j = 0; j < nb; ++j) step(t, j, kp);
      } else {
        for (int j = 0; j < nb; ++j)
          for (int kp = 0; kp < n_kp; ++kp) step(t, j, kp);
      }
    }
  };

  if (warp == ML_MMA_WARP) {
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t ring_u = __shfl_sync(0xffffffffu, sm0, 0);
    bool alive = true;
    uint32_t wslot = 0, wphase = 0;
    auto wait = [&](uint32_t bar, uint32_t parity) { if (alive) alive = mbar_wait(bar, parity & 1); };
    walk([&](int t, int j, int kp) {
      const uint32_t b = (uint32_t)(t * nb + j);  // number of the column block
      if (kp == 0 && b >= 3) wait(d_free + 8 * ((b - 3) % 6), (b - 3) / 6);
      const uint32_t gp = (uint32_t)(t * n_kpa + (shared_a ? kp : 2 * j + kp));
      const uint32_t abuf = 2 * (gp & 1);
      wait(a_ready + 8 * abuf, gp >> 1);
      wait(a_ready + 8 * (abuf + 1), gp >> 1);
      const uint32_t s_hi = wslot, p_hi = wphase;
      uint32_t s_lo = wslot + 1, p_lo = wphase;
      if (s_lo == ML_W_SLOTS) { s_lo = 0; ++p_lo; }
      wslot = s_lo + 1; wphase = p_lo;
      if (wslot == ML_W_SLOTS) { wslot = 0; ++wphase; }
      wait(w_ready + 8 * s_hi, p_hi);
      wait(w_ready + 8 * s_lo, p_lo);
      alive = __all_sync(0xffffffffu, alive);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d_tmem = tmem_u + 128u * (b % 3), ta = tmem_u + ML_A_BASE + 32u * abuf;
      if (elected) {
        const uint64_t dbh = umma_desc(ring_u + s_hi * TC_TILE_BYTES), dbl = umma_desc(ring_u + s_lo * TC_TILE_BYTES);
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const uint64_t adv = (uint64_t)(2 * (2 * ch + kk));
            const uint32_t t_hi = ta + 32 * ch + 8 * kk, t_lo = t_hi + 16;
            umma_bf16_ts(d_tmem, t_lo, dbh + adv, (kp > 0 || ch > 0 || kk > 0) ? 1u : 0u);
            umma_bf16_ts(d_tmem, t_hi, dbl + adv, 1u);
            umma_bf16_ts(d_tmem, t_hi, dbh + adv, 1u);
          }
        }
        mma_commit(w_done + 8 * s_hi);
        mma_commit(w_done + 8 * s_lo);
        if (!shared_a || j == nb - 1) { mma_commit(a_done + 8 * abuf); mma_commit(a_done + 8 * (abuf + 1)); }
        if (kp == n_kp - 1) mma_commit(d_full + 8 * (b % 6));
      }
      __syncwarp();
    });
    drain_mma(retired, elected);
  } else if (warp == ML_TMA_WARP) {
    pdl_sync();
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    const uint32_t ring_u = __shfl_sync(0xffffffffu, sm0, 0);
    bool alive = true;
    uint32_t n = 0, slot = 0, phase = 0;
    walk([&](int, int j, int kp) {
      if (!alive) return;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        if (n >= ML_W_SLOTS && alive) alive = mbar_wait(w_done + 8 * slot, (phase - 1) & 1);
        alive = __all_sync(0xffffffffu, alive);
        if (!alive) return;
        if (elected) {
          const uint32_t bar = w_ready + 8 * slot;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(TC_TILE_BYTES) : "memory");
          tma_load_2d(ring_u + slot * TC_TILE_BYTES, &maps.w[j0 + j][part], bar, 64 * kp, 0);
        }
        __syncwarp();
        ++n;
        if (++slot == ML_W_SLOTS) { slot = 0; ++phase; }
      }
    });
    drain_copies(w_ready, ML_W_SLOTS, n);
  } else if (warp == LN_SIDE_WARP) {
    // ---------------------------------------------------------------- gate / residual patches: lane e serves epilogue warp e
    pdl_sync();
    if (lane < 8) {
      const int q = (lane + 2) & 3;
      bool alive = true;
      uint32_t n = 0;
      for (int b = lane >> 2; b < n_tiles * nb; b += 2) {
        const int j = j0 + b % nb, row0 = (first_rt + (b / nb) * step_rt) * 128 + 32 * q;
        const mb_colblock& cb = d.blk[j];
        for (int c = 0; c < 4; ++c) {
#pragma unroll
          for (int what = 0; what < 2; ++what) {
            if (!(what == 0 ? (const void*)cb.gate : (const void*)cb.res) || !alive) continue;
            const uint32_t sl = n % SLOTS;
            if (n >= SLOTS) alive = mbar_wait(side_empty + 8 * (2 * lane + sl), (n / SLOTS - 1) & 1);
            if (!alive) continue;
            const uint32_t bar = side_full + 8 * (2 * lane + sl);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(ML_PATCH) : "memory");
            tma_load_2d(sm0 + ML_SIDE_OFF + (2 * lane + sl) * ML_PATCH, what == 0 ? &maps.gate[j] : &maps.res[j], bar, 32 * c, row0);
            ++n;
          }
        }
      }
      if constexpr (PAIR)
        drain_copies(side_full + 16 * lane, 1, n);
      else
        drain_copies(side_full + 16 * lane, 2, n);
    }
    __syncwarp();
  } else if (warp >= ML_EPI_WARP0) {
    pdl_sync();
    for (int i = tid - 32 * ML_EPI_WARP0; i < 1024; i += 256) {
      const mb_colblock& cb = d.blk[(i >> 7) & 3];
      const bool used = ((i >> 7) & 3) < nb_all;
      if (i < 512) cst[i] = used && cb.bias ? cb.bias[i & 127] : 0.f;
      else cst[i] = used && cb.res && cb.res_w ? cb.res_w[i & 127] : 1.f;
    }
    asm volatile("bar.sync 5, 256;" ::: "memory");  // the epilogue warps
    const int e = warp - ML_EPI_WARP0, q = warp & 3, grp = e >> 2;
    const uint32_t lane_q = tmem_base + ((uint32_t)(q * 32) << 16);
    const uint32_t side0 = sm0 + ML_SIDE_OFF + e * 2 * ML_PATCH, stage = sm0 + ML_STAGE_OFF + e * ML_PATCH;
    const uint32_t my_full = side_full + 16 * e, my_empty = side_empty + 16 * e;
    bool alive = true;
    uint32_t side_n = 0;
    auto wait = [&](uint32_t bar, uint32_t parity) {
      if (alive) alive = mbar_wait(bar, parity & 1);
      alive = __all_sync(0xffffffffu, alive);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    };
    auto with_patch = [&](auto f) {  // f(j, the row's 16-byte piece j) for the next side patch, which then goes back
      const uint32_t patch = side0 + side_n % SLOTS * ML_PATCH;
      wait(my_full + 8 * (side_n % SLOTS), side_n / SLOTS);
#pragma unroll
      for (int j = 0; j < 8; ++j) f(j, lds4(patch + lane * 128 + ((j ^ (lane & 7)) << 4)));
      __syncwarp();
      if (lane == 0) mbar_arrive(my_empty + 8 * (side_n % SLOTS));
      ++side_n;
    };
    for (int b = grp; b < n_tiles * nb; b += 2) {
      const int j = j0 + b % nb, row0 = (first_rt + (b / nb) * step_rt) * 128 + q * 32;
      const mb_colblock& cb = d.blk[j];
      const bool has_gate = cb.gate != nullptr, has_res = cb.res != nullptr, act = cb.out_act != 0, reduce = cb.mode != MB_OUT_STORE;
      const float sc = cb.out_scale;
      wait(d_full + 8 * (b % 6), (uint32_t)(b / 6));
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        float y[32];
        tmem_get(lane_q + 128u * (uint32_t)(b % 3) + 32u * c, y);
        if (c == 3) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(d_free + 8 * (b % 6));
        }
        const float4* const bias = reinterpret_cast<const float4*>(cst + 128 * j + 32 * c);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 v = bias[i];
          add4_to(y + 4 * i, v);
        }
        if (has_gate)
          with_patch([&](int i, const float4& v) {
            silu_grad4_to(y + 4 * i, v);
          });
        if (act) {
          silu_fast_all(y, y);
        }
        if (has_res) {
          const float4* const rw = reinterpret_cast<const float4*>(cst + 512 + 128 * j + 32 * c);
          with_patch([&](int i, const float4& v) {
            const float4 w = rw[i];
            fma4_to(y + 4 * i, v, w);
          });
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) apart(two(y[i], y[i + 1]) * two(sc, sc), y[i], y[i + 1]);
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the previous copy has left the patch
        __syncwarp();
        patch_put(stage, lane, y);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0 && alive && row0 < n_rows) {
          if (reduce) {  // one fp32 addition per element at the memory side; every row has one writer
            asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
                         :: "l"(reinterpret_cast<uint64_t>(&maps.out[j])), "r"(stage), "r"(32 * c), "r"(row0) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          } else {
            tma_store_2d(&maps.out[j], stage, 32 * c, row0);
          }
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    // ---------------------------------------------------------------- producers: lane quarter, K chunks of this warp's parity
    pdl_sync();
    const int pw = warp - ML_PROD_WARP0, parity = pw >> 2, quarter = warp & 3;
    const int lr = lane >> 3, lc = lane & 7;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t patch = sm0 + ML_CONV_OFF + pw * ML_PATCH, my_conv = conv_full + 8 * pw;
    const uint32_t put_even = lr * 128 + ((lc ^ lr) << 4), put_odd = lr * 128 + ((lc ^ (lr | 4)) << 4);
    bool alive = true;
    uint32_t g = (uint32_t)parity, conv_n = 0, conv_asked = 0;
    auto tile_row = [&](int t) { return (first_rt + t * step_rt) * 128 + quarter * 32; };
    auto request = [&](int t, int s, int k, bool stored) {
      if (!alive) return;
      ++conv_asked;
      if (lane == 0) {
        if (stored) to_async_proxy();  // the patch held gathered rows
        load_patch(&maps.src[shared_a ? s : j0 + s], patch, my_conv, 32 * (parity + 2 * k), tile_row(t));
      }
    };
    // PAIR: rows first and second of this lane's row in the current and the next tile, row numbers asked for two tiles ahead
    const uint32_t patch2 = sm0 + ML_SIDE_OFF + (2 * pw + 1) * ML_PATCH;
    int32_t first = 0, second = 0, first1 = 0, second1 = 0, first2 = 0;
    auto pair_row = [&](int t) {
      const int64_t r = t < n_tiles ? (int64_t)tile_row(t) + lane : 0;
      return d.blk[0].src[0].idx[r < n_rows ? r : n_rows - 1];
    };
    auto ask_pair = [&](int s, int k, int32_t r1, int32_t r2) {  // chunk k of segment s of both rows
      const mb_src& sr = segment(s);
      const float* const base = sr.ptr + sr.col + lc * 4 + 32 * (parity + 2 * k);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t at = ((i & 1) ? put_odd : put_even) + 512u * i;
        copy16(patch + at, base + (int64_t)__shfl_sync(0xffffffffu, r1, lr + 4 * i) * sr.ld);
        copy16(patch2 + at, base + (int64_t)__shfl_sync(0xffffffffu, r2, lr + 4 * i) * sr.ld);
      }
    };
    if constexpr (PAIR) {
      first = pair_row(0);
      first1 = pair_row(1);
      second = pair[first];
      ask_pair(0, 0, first, second);
    }
    if (!PAIR && segment(0).idx == nullptr) request(0, 0, 0, false);
    for (int t = 0; t < n_tiles; ++t) {
      if constexpr (PAIR) {
        second1 = pair[first1];
        first2 = pair_row(t + 2);
      }
      const int64_t row0 = tile_row(t);
      auto row_of = [&](int i) { const int64_t r = row0 + lr + 4 * i; return r < n_rows ? r : n_rows - 1; };
      for (int s = 0; s < n_seg; ++s) {
        const mb_src& sr = segment(s);
        const int32_t* const idx = sr.idx;
        const bool act = sr.act != 0;
#pragma unroll 1
        for (int k = 0; k < 2; ++k, g += 2) {
          if constexpr (PAIR) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
          } else if (!idx) {
            if (alive) alive = mbar_wait(my_conv, conv_n & 1);
            alive = __all_sync(0xffffffffu, alive);
            ++conv_n;
          } else {
            const float* const base = sr.ptr + sr.col + lc * 4 + 32 * (parity + 2 * k);
            float4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = ld4(base + (int64_t)idx[row_of(i)] * sr.ld);
#pragma unroll
            for (int i = 0; i < 8; ++i) sts4(patch + ((i & 1) ? put_odd : put_even) + 512u * i, v[i].x, v[i].y, v[i].z, v[i].w);
            __syncwarp();
          }
          float x[32];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 v = lds4(patch + lane * 128 + ((i ^ (lane & 7)) << 4));
            x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
          }
          const int s2 = k == 0 ? s : (s + 1 < n_seg ? s + 1 : 0), t2 = k == 1 && s + 1 == n_seg ? t + 1 : t;  // the chunk after this one
          if constexpr (PAIR) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 v = lds4(patch2 + lane * 128 + ((i ^ (lane & 7)) << 4));
              add4_to(x + 4 * i, v);
            }
            __syncwarp();  // every lane has read: the next chunk's copies may be asked for
            if (t2 < n_tiles) ask_pair(s2, k ^ 1, t2 == t ? first : first1, t2 == t ? second : second1);
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
          if (!PAIR && t2 < n_tiles && segment(s2).idx == nullptr) request(t2, s2, k ^ 1, idx != nullptr);
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(a_ready + 8 * ab);
        }
      }
      if constexpr (PAIR) { first = first1; second = second1; first1 = first2; }
    }
    if (!alive) drain_copies(my_conv, 1, conv_asked);  // (otherwise it has used all that it asked for)
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == ML_MMA_WARP) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(PS_TMEM_COLS) : "memory");
  }
}
