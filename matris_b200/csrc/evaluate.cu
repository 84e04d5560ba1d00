// Whole-model driver: queues every kernel of an evaluation (graph tensors -> energies, forces, stresses, moments) from
// one host call.
//
// What bounds a small system is the host: an evaluation is 440 - 640 launches, and from an interpreter each costs about
// 20 us (descriptor packing, foreign-function call, tensor allocation, autograd bookkeeping).  Queued from here a launch costs
// 2 - 3 us: when they were 600 - 800, 4 atoms 13.2 -> 9.2 ms, bound by the device ever since.
//
// Memory is handed out from two stacks: inputs of the sub-blocks (always needed by the backward pass) and temporaries on the
// bottom one, internals of the layers that keep them on the top one.  The backward pass pops both in reverse order.  A small
// evaluation takes one workspace of the caller's, used from both ends; a large one (whose workspace could approach the whole
// device and would fragment the caller's allocator) asks the caller's allocator for every buffer.  Run dry, the same code
// only counts, which is how a workspace is sized and how many layers keep their internals is decided: the counts cannot
// disagree with the run.
#include <stdio.h>
#include <string.h>
#include <array>
#include <exception>
#include <initializer_list>
#include <mutex>
#include <vector>
#include "common.cuh"

namespace mb {

// ------------------------------------------------------------------ small kernels
// Per structure: e = (sum of its atoms' energies) / n + sum_z (n_z / n) table[z]  (no division when the model is
// extensive); one warp per structure.  The composition is counted exactly in shared memory (int), then folded in float32
// like the reference's composition-row x table product (matris/model/reference_energy.py:34-55).
constexpr int FIN_WARPS = 4, FIN_SPECIES = 128;
__global__ void k_energy_finish(int n_struct, const int32_t* __restrict__ atom_ptr, const float* __restrict__ e_atom,
                                const int32_t* __restrict__ numbers, const float* __restrict__ table, int n_species,
                                int intensive, float* __restrict__ e, float* __restrict__ ref, int32_t* __restrict__ apg) {
  pdl_sync();
  __shared__ int count[FIN_WARPS][FIN_SPECIES];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = blockIdx.x * FIN_WARPS + w;
  if (b >= n_struct) return;
  const int a0 = atom_ptr[b], a1 = atom_ptr[b + 1];
  for (int z = lane; z < FIN_SPECIES; z += 32) count[w][z] = 0;
  __syncwarp();
  float s = 0.f;
  for (int i = a0 + lane; i < a1; i += 32) {
    s += e_atom[i];
    const int z = numbers[i] - 1;
    if (table && z >= 0 && z < n_species) atomicAdd(&count[w][z], 1);
  }
  __syncwarp();
  s = warp_sum(s);
  const float n = (float)(a1 - a0);
  float r = 0.f;
  if (table)
    for (int z = lane; z < n_species; z += 32) {
      const float c = (float)count[w][z];
      r = fmaf(intensive ? c / n : c, table[z], r);
    }
  r = warp_sum(r);
  if (lane == 0) {
    e[b] = (intensive ? s / n : s) + r;
    if (ref) ref[b] = r;
    if (apg) apg[b] = a1 - a0;
  }
}

// forces = - dE/dr ; stress in GPa = dE/dstrain * (GPa per eV/A^3 / volume)
__global__ void k_force_stress_finish(int n_atoms, int n_struct, const float* __restrict__ dcart,
                                      const float* __restrict__ dstrain, const float* __restrict__ volume,
                                      float* __restrict__ f, float* __restrict__ s) {
  pdl_sync();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (f && i < 3 * (int64_t)n_atoms) f[i] = -dcart[i];
  if (s && i < 9 * (int64_t)n_struct) s[i] = dstrain[i] * (160.21766208f / volume[i / 9]);
}

// a memset that joins the chain of programmatic launches (the copy engine's would end it before and after): n 4-byte words
__global__ void k_zero(size_t n, float* __restrict__ p) {
  pdl_sync();
  const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i + 4 <= n) *reinterpret_cast<float4*>(p + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  else for (size_t k = i; k < n; ++k) p[k] = 0.f;
}

// ------------------------------------------------------------------ instrumentation
struct OpTimes {
  bool on = false;
  struct Rec { mb_op_record r; cudaEvent_t a, b; };
  std::vector<Rec> recs;
};
static OpTimes g_times;  // a measuring aid for one thread at a time

// ------------------------------------------------------------------ memory
struct Arena {
  enum Mode { DRY, BUFFER, CALLBACK };
  struct Piece { void* p; size_t bytes; };
  Mode mode = DRY;
  char* base = nullptr;
  size_t cap = 0, lo = 0, hi = 0, peak = 0;
  bool failed = false;
  mb_alloc_fn alloc = nullptr;
  mb_free_fn release = nullptr;
  std::vector<Piece> low, high;
  ~Arena() { drop(low, lo, 0); drop(high, hi, 0); }

  float* take(std::vector<Piece>& stack, size_t& used, size_t floats, bool from_top) {
    // Large buffers in steps of 1/32 of their power of two: successive batches of about the same size then ask the
    // allocator for the same sizes, and find their predecessors' blocks.
    size_t step = 256;
    while (step * 64 <= floats * 4) step *= 2;
    const size_t bytes = (floats * 4 + step - 1) / step * step;
    stack.push_back({nullptr, bytes});  // (may throw: before anything is taken)
    used += bytes;
    if (lo + hi > peak) peak = lo + hi;
    void* p = nullptr;
    if (mode == DRY) p = reinterpret_cast<void*>(256);  // not NULL, never dereferenced
    else if (mode == BUFFER) p = lo + hi > cap ? nullptr : base + (from_top ? cap - hi : lo - bytes);
    else if (!failed) p = bytes ? alloc(bytes) : reinterpret_cast<void*>(256);
    if (!p) failed = true;
    stack.back() = {p, bytes};
    return static_cast<float*>(p);
  }
  void drop(std::vector<Piece>& stack, size_t& used, size_t count) {
    while (stack.size() > count) {
      const Piece t = stack.back();
      stack.pop_back();
      used -= t.bytes;
      if (mode == CALLBACK && t.p && t.bytes) release(t.p);
    }
  }
  float* bottom(size_t floats) { return take(low, lo, floats, false); }
  float* top(size_t floats) { return take(high, hi, floats, true); }
};

// ------------------------------------------------------------------ side streams
// Two more streams for work that does not feed the next kernel of the caller's stream.  A small system is bound by the chain of its
// launches, most of which leave most SMs idle: off the chain go a layer's centre and node tables, the logits, the envelopes and
// the other of two feed-forward blocks, in the backward pass the node sums beside the edge gradients.  Device time of an evaluation:
// 32 atoms 6.5 -> 5.5 ms, 256 atoms 10.4 -> 9.4; 16,000 atoms 624 -> 608 (tails of one launch filled by another), so for all sizes.
// Taken from a pool for one call and given back when its work is queued (a later user of the same streams queues behind it); the
// pool keeps no more than eight sets.
struct Side {
  int device = -1;
  cudaStream_t st[2] = {};
  cudaEvent_t ev = nullptr;
};
static std::mutex g_side_mutex;
static std::vector<Side> g_side_pool;

static void side_free(Side& s) {
  for (cudaStream_t t : s.st)
    if (t) cudaStreamDestroy(t);  // (work still queued there runs to its end)
  if (s.ev) cudaEventDestroy(s.ev);
}
static bool side_take(Side& s) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  {
    std::lock_guard<std::mutex> lock(g_side_mutex);
    for (size_t i = 0; i < g_side_pool.size(); ++i)
      if (g_side_pool[i].device == dev) {
        s = g_side_pool[i];
        g_side_pool.erase(g_side_pool.begin() + i);
        return true;
      }
  }
  s.device = dev;
  auto failed = [&] {  // the evaluation goes on without: its first launch must not find this error as its own
    side_free(s);
    cudaGetLastError();
    return false;
  };
  for (cudaStream_t& t : s.st)
    if (cudaStreamCreateWithFlags(&t, cudaStreamNonBlocking) != cudaSuccess) return failed();
  if (cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming) != cudaSuccess) return failed();
  return true;
}
static void side_give(Side& s) {
  {
    std::lock_guard<std::mutex> lock(g_side_mutex);
    if (g_side_pool.size() < 8) {
      g_side_pool.push_back(s);
      return;
    }
  }
  side_free(s);
}

struct Run {
  Arena ar;
  cudaStream_t st = nullptr;
  Side* sides = nullptr;  // NULL: everything on the caller's stream
  bool pending[2] = {};
  int on = 0;             // 0: the caller's stream, 1 + k: side stream k
  bool behind[3] = {};    // the last thing queued there is a wait for another stream's event
  bool queued[3] = {};    // this evaluation has launched something there

  // f's launches on side stream k, after everything queued on the caller's stream so far.  The buffers they touch must live, and
  // must not be written or (where f writes) read on the caller's stream, until join(k).
  template <typename F> void side(int k, F f) {
    if (!sides || !go()) {
      f();
      return;
    }
    const cudaStream_t main = st;
    after(1 + k, sides->st[k], main);
    st = sides->st[k]; on = 1 + k;
    f();
    st = main; on = 0;
    pending[k] = true;
  }
  void join(int k) {
    if (!pending[k]) return;
    pending[k] = false;
    after(0, st, sides->st[k]);
  }
  void after(int which, cudaStream_t later, cudaStream_t earlier) {
    if (cudaEventRecord(sides->ev, earlier) != cudaSuccess || cudaStreamWaitEvent(later, sides->ev, 0) != cudaSuccess)
      rc = rc == MB_OK ? MB_ERR_CUDA : rc;
    behind[which] = true;
  }
  int rc = MB_OK, launches = 0;
  bool scratch = false;  // the contraction mode composes a gated MLP from separate launches, which need z1 / z2

  bool go() {
    if (ar.failed && rc == MB_OK) rc = MB_ERR_CAPACITY;
    return ar.mode != Arena::DRY && rc == MB_OK;
  }
  template <typename F> void op(const char* name, F f, double flops = 0, double bytes = 0, int64_t rows = 0, int k = 0,
                                int n = 0, int fused = 0) {
    if (!go()) return;
    ++launches;
    if (!g_times.on) {
      launch_after_event = behind[on];
      weights_settled = behind[on] || queued[on];
      rc = f();
      weights_settled = false;
      queued[on] = true;
      behind[on] = launch_after_event;  // (what launches nothing leaves it)
      launch_after_event = false;
      return;
    }
    OpTimes::Rec rec{};
    snprintf(rec.r.name, sizeof(rec.r.name), "%s", name);
    rec.r.flops = flops; rec.r.bytes = bytes; rec.r.rows = rows; rec.r.k = k; rec.r.n = n; rec.r.fused = fused;
    if (cudaEventCreate(&rec.a) != cudaSuccess || cudaEventCreate(&rec.b) != cudaSuccess) { rc = MB_ERR_CUDA; return; }
    cudaEventRecord(rec.a, st);
    rc = f();
    cudaEventRecord(rec.b, st);
    g_times.recs.push_back(rec);
  }
  void zero(float* p, size_t bytes) {
    if (bytes == 0) return;
    op("memset", [&] {
      launch(k_zero, (unsigned)((bytes / 16 + 256) / 256), 256, 0, st, bytes / 4, p);
      MB_LAUNCH_CHECK("k_zero");
      return (int)MB_OK;
    });
  }
};
#define MB_OP(name, ...) R.op(#name, [&] { return name(__VA_ARGS__, R.st); })

// releases the bottom stack at the end of a scope
struct Scope {
  Run& R;
  size_t mark;
  bool open = true;
  explicit Scope(Run& r) : R(r), mark(r.ar.low.size()) {}
  ~Scope() { if (open) close(); }
  void close() {
    open = false;
    R.ar.drop(R.ar.low, R.ar.lo, mark);
  }
};

// ------------------------------------------------------------------ contractions
static inline mb_src src(const float* p, const int32_t* idx = nullptr, int col = 0, int64_t ld = 128, int act = 0) {
  mb_src s;
  s.ptr = p; s.idx = idx; s.ld = ld; s.col = col; s.act = act;
  return s;
}

struct Gemm {
  mb_gemm_desc d;
  explicit Gemm(int64_t rows) { memset(&d, 0, sizeof(d)); d.n_rows = rows; }
  mb_colblock& block(std::initializer_list<mb_src> srcs, const mb_weight& w, int w_row, float* out, int64_t ld_out,
                     int col_out = 0, const int32_t* out_idx = nullptr, int mode = MB_OUT_STORE) {
    mb_colblock& b = d.blk[d.n_blocks++];
    for (const mb_src& s : srcs) b.src[b.n_src++] = s;
    const int64_t o = w.ldw * w_row;
    b.W = w.W + o; b.W_hi = w.W_hi ? w.W_hi + o : nullptr; b.W_lo = w.W_lo ? w.W_lo + o : nullptr;
    b.W_hi16 = w.W_hi16 ? w.W_hi16 + o : nullptr; b.W_lo16 = w.W_lo16 ? w.W_lo16 + o : nullptr;
    b.ldw = w.ldw;
    b.out = out; b.ld_out = ld_out; b.col_out = col_out; b.out_idx = out_idx; b.mode = mode; b.out_scale = 1.f;
    return b;
  }
  void run(Run& R, const int32_t* pair = nullptr) {
    if (d.n_rows == 0 || d.n_blocks == 0) return;
    double flops = 0, bytes = 4.0 * d.n_rows * 128 * ((pair ? 2 : 1) * d.blk[0].n_src + d.n_blocks);
    for (int j = 0; j < d.n_blocks; ++j) {
      flops += 2.0 * d.n_rows * 128 * 128 * d.blk[j].n_src;
      bytes += 4.0 * d.n_rows * 128 * ((d.blk[j].gate != nullptr) + (d.blk[j].res != nullptr));
    }
    R.op("mb_gemm", [&] { return pair ? pair_linear(&d, pair, R.st) : mb_gemm(&d, R.st); }, flops, bytes, d.n_rows, 128 * d.blk[0].n_src, 128 * d.n_blocks);
  }
};

// Independent contractions of few rows as one launch, without the 4 - 9 us that a side stream's fork and join add to the chain;
// false: nothing done, they do not all run side by side in one
static bool together(Run& R, std::initializer_list<Gemm*> all) {
  const mb_gemm_desc* d[4];
  int n = 0;
  double flops = 0, bytes = 0;
  for (Gemm* g : all) {
    if (g->d.n_rows == 0 || g->d.n_blocks == 0) continue;
    d[n++] = &g->d;
    for (int j = 0; j < g->d.n_blocks; ++j) flops += 2.0 * g->d.n_rows * 128 * 128 * g->d.blk[j].n_src;
    bytes += 4.0 * g->d.n_rows * 128 * (g->d.blk[0].n_src + g->d.n_blocks);
  }
  if (!R.go() || n < 2 || !few_linears_fit(d, n)) return false;
  R.op("mb_gemm", [&] { return few_linears(d, n, R.st); }, flops, bytes, d[0]->n_rows, 128 * d[0]->blk[0].n_src, 128 * d[0]->n_blocks);
  return true;
}

// y [rows, 128 nb] = epilogue(x [rows, 128 ns] W^T), ns = k / 128, nb = n_out / 128
struct LinearOpt {
  const float* bias = nullptr; int out_act = 0, in_act = 0; const float* gate = nullptr; float scale = 1.f;
  const int32_t* idx = nullptr;
};
static Gemm dense(int64_t rows, const float* x, const mb_weight& w, int n_out, int k, float* out, const LinearOpt& o = LinearOpt()) {
  const int ns = k / 128, nb = n_out / 128;
  Gemm g(rows);
  for (int j = 0; j < nb; ++j) {
    mb_colblock& b = g.block({}, w, 128 * j, out, n_out, 128 * j);
    for (int s = 0; s < ns; ++s) b.src[b.n_src++] = src(x, o.idx, 128 * s, k, o.in_act);
    b.bias = o.bias ? o.bias + 128 * j : nullptr;
    b.out_act = o.out_act;
    if (o.gate) { b.gate = o.gate; b.ld_gate = n_out; b.col_gate = 128 * j; }
    b.out_scale = o.scale;
  }
  return g;
}
static void linear(Run& R, int64_t rows, const float* x, const mb_weight& w, int n_out, int k, float* out,
                   const LinearOpt& o = LinearOpt()) {
  dense(rows, x, w, n_out, k, out, o).run(R);
}

static void fill_mlp(mb_gated_mlp& m, int64_t rows, std::initializer_list<mb_src> srcs, const mb_weight& w1,
                     const mb_weight& w2, const float* b1, const float* b2) {
  memset(&m, 0, sizeof(m));
  m.n_rows = rows;
  for (const mb_src& s : srcs) m.src[m.n_src++] = s;
  m.W1 = w1.W; m.W1_hi = w1.W_hi; m.W1_lo = w1.W_lo; m.W1_hi16 = w1.W_hi16; m.W1_lo16 = w1.W_lo16; m.ldw1 = w1.ldw;
  m.W2 = w2.W; m.W2_hi = w2.W_hi; m.W2_lo = w2.W_lo; m.W2_hi16 = w2.W_hi16; m.W2_lo16 = w2.W_lo16; m.ldw2 = w2.ldw;
  m.b1 = b1; m.b2 = b2;
}

static void run_mlp(Run& R, const mb_gated_mlp& m) {
  if (m.n_rows == 0) return;
  const int n = m.kind == MB_MLP_PLAIN ? 128 : 256;
  const double flops = 2.0 * m.n_rows * n * 128 * (m.n_src + 1);
  const double bytes = 4.0 * m.n_rows * 128 * (m.n_src + (m.z1 ? n / 128 : 0) + (m.z2 ? n / 128 : 0) + (m.h != nullptr) +
                                               2 * (m.out2 != nullptr));
  R.op("mb_gated_mlp_fwd", [&] { return mb_gated_mlp_fwd(&m, R.st); }, flops, bytes, m.n_rows, 128 * m.n_src, n, 1);
}

// ------------------------------------------------------------------ update blocks
// Forward of an update block.  z1 / z2 (width 256 gated, 128 plain MLP) may be NULL when nothing needs them later; h and
// out2 = h + res_w * res are optional.
static int update_width(const mb_update& p) { return p.kind == MB_UPDATE_MLP ? 128 : 256; }
static void update_fwd(Run& R, const mb_update& p, int64_t rows, std::initializer_list<mb_src> srcs, float* z1, float* z2,
                       float* h, const float* res, const float* res_w, float* out2) {
  Scope sc(R);
  if (p.kind == MB_UPDATE_MLP) {
    if (!z1) z1 = R.ar.bottom(rows * 128);
    if (!z2) z2 = R.ar.bottom(rows * 128);
    Gemm a(rows), b(rows);
    a.block(srcs, p.w1, 0, z1, 128).bias = p.b1;
    a.run(R);
    b.block({src(z1, nullptr, 0, 128, 1)}, p.w2, 0, z2, 128).bias = p.b2;
    b.run(R);
    if (h) MB_OP(mb_rmsnorm_fwd, rows, z2, p.nc, h);
    if (out2) {
      MB_OP(mb_rmsnorm_fwd, rows, z2, p.nc, out2);
      MB_OP(mb_scale_rows, rows, res, res_w, out2, 1);
    }
    return;
  }
  if (R.scratch) {
    if (!z1) z1 = R.ar.bottom(rows * 256);
    if (!z2) z2 = R.ar.bottom(rows * 256);
  }
  mb_gated_mlp m;
  fill_mlp(m, rows, srcs, p.w1, p.w2, p.b1, p.b2);
  m.norm_core = p.nc; m.norm_gate = p.ng;
  m.z1 = z1; m.ld_z1 = 256; m.z2 = z2; m.ld_z2 = 256; m.h = h; m.ld_h = 128;
  m.res = out2 ? res : nullptr; m.res_w = out2 ? res_w : nullptr; m.ld_res = 128; m.out2 = out2; m.ld_out2 = 128;
  run_mlp(R, m);
}

// Edge update of a gated kind: layer 1 from tables of finished sums per node (P = node [Wt | Ws]^T), per bond (atom graph:
// bonds We^T, the directed rows only gather) and per centre atom (line-graph refinement).  With `logits` the attention logits
// of the edge features come out of the same launch as the bond table (atom graph) or of one of their own.
static void edge_update_fwd(Run& R, const mb_update& p, const mb_row_graph& g, const float* node, const float* edge,
                            const float* ctr_feat, const mb_weight* wst, float* logits, float* z1, float* z2, float* h,
                            const float* res_w, float* out2) {
  if (p.kind == MB_UPDATE_MLP) {
    if (g.is_atom || !ctr_feat)
      update_fwd(R, p, g.n_rows, {src(edge, g.emap), src(node, g.tgt), src(node, g.src)}, z1, z2, h, edge, res_w, out2);
    else
      update_fwd(R, p, g.n_rows, {src(edge), src(ctr_feat, g.ctr), src(node, g.tgt), src(node, g.src)}, z1, z2, h, edge, res_w,
                 out2);
    if (logits) linear(R, g.n_edge_rows, edge, *wst, 256, 128, logits);
    return;
  }
  Scope sc(R);
  float* P = R.ar.bottom((size_t)g.n_nodes * 512);
  float* Pc = ctr_feat ? R.ar.bottom((size_t)g.n_ctr * 256) : nullptr;
  float* Pe = g.is_atom ? R.ar.bottom((size_t)g.n_edge_rows * 256) : nullptr;
  if (R.scratch) {
    if (!z1) z1 = R.ar.bottom((size_t)g.n_rows * 256);
    if (!z2) z2 = R.ar.bottom((size_t)g.n_rows * 256);
  }
  Gemm nodes = dense(g.n_nodes, node, p.wts, 512, 128, P), centres(0);
  if (Pc) centres = dense(g.n_ctr, ctr_feat, p.wc, 256, 128, Pc);
  Gemm e(g.n_edge_rows);
  if (Pe)
    for (int j = 0; j < 2; ++j) e.block({src(edge)}, p.we, 128 * j, Pe, 256, 128 * j);
  if (logits)
    for (int j = 0; j < 2; ++j) e.block({src(edge)}, *wst, 128 * j, logits, 256, 128 * j);
  if (!together(R, {&e, &nodes, &centres})) {
    if (Pc) R.side(0, [&] { centres.run(R); });
    if (g.is_atom) {
      R.side(0, [&] { nodes.run(R); });
      e.run(R);
      R.join(0);
    } else {  // e holds the logits at most, which the caller waits for
      if (e.d.n_blocks) R.side(0, [&] { e.run(R); });
      nodes.run(R);
      if (Pc) R.join(0);
    }
  }
  mb_gated_mlp m;
  if (g.is_atom) fill_mlp(m, g.n_rows, {}, p.we, p.w2, p.b1, p.b2);
  else fill_mlp(m, g.n_rows, {src(edge)}, p.we, p.w2, p.b1, p.b2);
  m.norm_core = p.nc; m.norm_gate = p.ng;
  m.z1 = z1; m.ld_z1 = 256; m.z2 = z2; m.ld_z2 = 256; m.h = h; m.ld_h = 128;
  m.res = out2 ? edge : nullptr; m.res_w = out2 ? res_w : nullptr; m.ld_res = 128; m.out2 = out2; m.ld_out2 = 128;
  auto add = [&](const float* t, const int32_t* idx, int64_t ld) { m.add[m.n_add++] = mb_add{t, idx, ld}; };
  add(P, g.tgt, 512);
  add(P + 256, g.src, 512);
  if (Pe) add(Pe, g.emap, 256);
  if (Pc) add(Pc, g.ctr, 256);
  run_mlp(R, m);
}

// The row gradient's launch where the few-row product does not form it itself (same expressions): dz2 from rg.
static int row_grad(const RowGrad& g, int64_t rows, float* dz2, cudaStream_t st) {
  if (g.kind == 1)
    return mb_seg_attn_bwd(rows, g.tgt, g.src, g.idx_stride, g.emap, g.logits, g.h, g.agg_t, g.agg_s, g.stats, g.dagg_t, g.dagg_s,
                           g.dh_in, g.dh_map, g.dh_scale, nullptr, g.dlogits, g.z2, g.norm_core, g.norm_gate, dz2, st);
  return mb_seg_smooth_sum_bwd_rows(rows, g.tgt, g.src, g.idx_stride, g.emap, g.env, g.dagg, const_cast<float*>(g.dh_in),
                                    g.dh_in ? 1 : 0, g.z2, g.norm_core, g.norm_gate, dz2, st);
}

// Backward of the same from the rows' gradient rg on (its dlogits where given): d_edge = ... + edge_w * edge_res, d_node (+)= ... + node_w * node_res, the centre
// atoms' gradient is accumulated into d_ctr.
static void edge_update_bwd(Run& R, const mb_update& p, const mb_row_graph& g, const float* z1, const RowGrad& rg, float* dz2,
                            const mb_weight* w_log, const float* edge_res, const float* edge_w,
                            float* d_edge, const float* node_res, const float* node_w, float* d_node, float* d_ctr) {
  Scope sc(R);
  float* dz1 = R.ar.bottom((size_t)g.n_rows * 256);
  float* dP = R.ar.bottom((size_t)g.n_nodes * 512);
  float* dPc = d_ctr ? R.ar.bottom((size_t)g.n_ctr * 256) : nullptr;
  float* const dlogits = rg.dlogits;
  const bool few = R.go() && few_row_bwd_fits(g.n_rows, 1, !g.is_atom && dlogits);
  RowBwd b{};
  if (few) {
    b.n_rows = g.n_rows; b.g = rg; b.w2t = p.w2t; b.z1 = z1; b.dz1 = dz1;
    if (!g.is_atom) {
      b.g.dlogits = nullptr;  // used on the way
      b.w1t = p.wet; b.n_out = 1; b.out[0] = d_edge; b.res = edge_res; b.res_w = edge_w;
      if (dlogits) b.w3t = *w_log;
      b.zero = dPc; b.n_zero = dPc ? (int64_t)g.n_ctr * 256 : 0;
    }
    const double k = b.n_out ? (dlogits ? 768 : 512) : 256;
    R.op(dlogits ? "mb_attn_mlp_bwd" : "mb_smooth_mlp_bwd", [&] { return few_row_bwd(b, R.st); }, 2.0 * g.n_rows * 128 * k,
         4.0 * g.n_rows * 128 * 8, g.n_rows, 256, 256, 1);
  } else {
    R.op(rg.kind == 1 ? "mb_seg_attn_bwd" : "mb_seg_smooth_sum_bwd_rows", [&] { return row_grad(rg, g.n_rows, dz2, R.st); });
    if (dPc) R.zero(dPc, (size_t)g.n_ctr * 1024);
  }
  auto node_sums = [&] {
    MB_OP(mb_seg_sum, (int32_t)g.n_nodes, g.n_rows, g.tgt_ptr, g.src_ptr, g.src_perm, d_ctr ? g.ctr : nullptr, dz1, dP, dPc);
  };
  Gemm n(g.n_nodes);
  {
    mb_colblock& b = n.block({src(dP, nullptr, 0, 512), src(dP, nullptr, 128, 512), src(dP, nullptr, 256, 512),
                              src(dP, nullptr, 384, 512)}, p.wtst, 0, d_node, 128, 0, nullptr, node_res ? MB_OUT_STORE : MB_OUT_ADD);
    b.res = node_res; b.res_w = node_w; b.ld_res = 128;
  }
  if (g.is_atom) {
    if (!few) {
      Gemm a(g.n_rows);
      for (int j = 0; j < 2; ++j) {
        mb_colblock& b = a.block({src(dz2, nullptr, 128 * j, 256)}, p.w2t, 128 * j, dz1, 256, 128 * j);
        b.gate = z1; b.ld_gate = 256; b.col_gate = 128 * j;
      }
      a.run(R);
    }
    R.side(0, [&] {
      node_sums();
      n.run(R);
    });
    // the sums, where a launch of its own forms them, in the place of dz2, which has been read by then ([n_rows, 256] = [n_edge_rows, 512])
    float* const pair = 2 * g.n_edge_rows <= g.n_rows ? dz2 : R.ar.bottom((size_t)g.n_edge_rows * 512);
    Gemm e(g.n_edge_rows);
    mb_colblock& b = e.block({}, dlogits ? *w_log : p.wet, 0, d_edge, 128);
    b.res = edge_res; b.res_w = edge_w; b.ld_res = 128;
    b.n_src = dlogits ? 4 : 2;  // the sums of dz1 (core, gate) and of dlogits, formed on the way
    for (int j = 0; j < b.n_src; ++j) b.src[j] = src(j < 2 ? dz1 : dlogits, g.u2d, 128 * (j & 1), 256);
    const bool pairs = pair_linear_fits(&e.d);
    if (!pairs) {  // contraction modes other than the default, weights that are not aligned to 32 bytes
      const int ld = dlogits ? 512 : 256;
      MB_OP(mb_pair_sum, (int32_t)g.n_edge_rows, g.u2d, g.rev, dz1, dlogits, pair);
      for (int j = 0; j < b.n_src; ++j) b.src[j] = src(pair, nullptr, 128 * j, ld);
    }
    e.run(R, pairs ? g.rev : nullptr);
  } else if (!few) {
    mb_mlp_bwd m;
    memset(&m, 0, sizeof(m));
    m.n_rows = g.n_rows; m.kind = MB_MLP_GATED;
    m.dy = src(dz2, nullptr, 0, 256);
    m.W2t = p.w2t; m.W1t = p.wet;
    m.z1 = z1; m.ld_z1 = 256; m.dz1 = dz1; m.ld_dz1 = 256; m.dx = d_edge; m.ld_dx = 128;
    m.res = edge_res; m.res_w = edge_w; m.ld_res = 128;
    if (dlogits) {
      m.n_ext = 2;
      for (int j = 0; j < 2; ++j) m.ext[j] = src(dlogits, nullptr, 128 * j, 256);
      m.W3t = *w_log;
    }
    const double k = dlogits ? 768 : 512;
    R.op("mb_mlp_bwd_data", [&] { return mb_mlp_bwd_data(&m, R.st); }, 2.0 * g.n_rows * 128 * k,
         4.0 * g.n_rows * 128 * (7 + (edge_res != nullptr) + (dlogits ? 2 : 0)), g.n_rows, 256, 256, 1);
  }
  if (!g.is_atom) {
    node_sums();
    Gemm c(g.n_ctr);
    if (dPc) c.block({src(dPc, nullptr, 0, 256), src(dPc, nullptr, 128, 256)}, p.wct, 0, d_ctr, 128, 0, nullptr, MB_OUT_ADD);
    if (!together(R, {&n, &c})) {
      if (dPc) R.side(0, [&] { c.run(R); });
      n.run(R);
    }
  }
  R.join(0);
}

struct Dest {  // where the gradient of one 128-wide K segment goes
  float* t; const int32_t* idx; int mode; const float* res; const float* res_w;
};
// Backward: dh [rows,128] in (or dz2 [rows,256], where its producer applied the gated tail's adjoint already).
static void update_bwd(Run& R, const mb_update& p, int64_t rows, const float* z1, const float* z2, const float* dh,
                       const float* dz2, std::initializer_list<Dest> dests) {
  Scope sc(R);
  Gemm out(rows);
  if (p.kind == MB_UPDATE_MLP) {
    float* dy = R.ar.bottom(rows * 128);
    float* da = R.ar.bottom(rows * 128);
    MB_OP(mb_rmsnorm_bwd, rows, z2, p.nc, dh, dy);
    LinearOpt o;
    o.gate = z1;
    linear(R, rows, dy, p.w2t, 128, 128, da, o);
    int c = 0;
    for (const Dest& d : dests) {
      mb_colblock& b = out.block({src(da)}, p.w1t, 128 * c++, d.t, 128, 0, d.idx, d.mode);
      b.res = d.res; b.res_w = d.res_w; b.ld_res = 128;
    }
    out.run(R);
    return;
  }
  float* const t = dz2 ? nullptr : R.ar.bottom(rows * 256);
  float* dz1 = R.ar.bottom(rows * 256);
  bool plain = dests.size() <= 3;  // outputs at their own rows, a residual on the first at most
  for (const Dest& d : dests) plain = plain && !d.idx && d.mode == MB_OUT_STORE && (!d.res || &d == dests.begin());
  if (!dz2 && plain && R.go() && few_row_bwd_fits(rows, (int)dests.size(), false)) {
    RowBwd b{};
    b.n_rows = rows; b.w2t = p.w2t; b.w1t = p.w1t; b.z1 = z1;
    b.g.dh_in = dh; b.g.z2 = z2; b.g.norm_core = p.nc; b.g.norm_gate = p.ng;
    for (const Dest& d : dests) b.out[b.n_out++] = d.t;
    b.res = dests.begin()->res; b.res_w = dests.begin()->res_w;
    R.op("mb_node_mlp_bwd", [&] { return few_row_bwd(b, R.st); }, 2.0 * rows * 256 * (128 + 128 * b.n_out), 4.0 * rows * 128 * (6 + b.n_out),
         rows, 256, 128 * b.n_out, 1);
    return;
  }
  if (!dz2) {
    MB_OP(mb_gate_bwd, rows, z2, p.nc, p.ng, dh, t);
    dz2 = t;
  }
  Gemm g(rows);
  for (int j = 0; j < 2; ++j) {
    mb_colblock& b = g.block({src(dz2, nullptr, 128 * j, 256)}, p.w2t, 128 * j, dz1, 256, 128 * j);
    b.gate = z1; b.ld_gate = 256; b.col_gate = 128 * j;
  }
  g.run(R);
  int c = 0;
  for (const Dest& d : dests) {
    mb_colblock& b = out.block({src(dz1, nullptr, 0, 256), src(dz1, nullptr, 128, 256)}, p.w1t, 128 * c++, d.t, 128, 0, d.idx,
                               d.mode);
    b.res = d.res; b.res_w = d.res_w; b.ld_res = 128;
  }
  out.run(R);
}

static void ffn_fwd(Run& R, const mb_ffn& p, int64_t rows, const float* x, float* z1, float* y, const float* res,
                    const float* res_w, float* out2) {
  Scope sc(R);
  if (R.scratch && !z1) z1 = R.ar.bottom(rows * 128);
  mb_gated_mlp m;
  fill_mlp(m, rows, {src(x)}, p.w1, p.w2, p.b1, p.b2);
  m.kind = MB_MLP_PLAIN;
  m.z1 = z1; m.ld_z1 = 128; m.h = y; m.ld_h = 128;
  m.res = out2 ? res : nullptr; m.res_w = out2 ? res_w : nullptr; m.ld_res = 128; m.out2 = out2; m.ld_out2 = 128;
  run_mlp(R, m);
}

// dx = scale * ((dy W2) * silu'(z1)) W1 ; dy optionally gathered
static mb_mlp_bwd ffn_grad(const mb_ffn& p, int64_t rows, const float* dy, const int32_t* idx, float scale, const float* z1, float* dx) {
  mb_mlp_bwd m;
  memset(&m, 0, sizeof(m));
  m.n_rows = rows; m.kind = MB_MLP_PLAIN;
  m.dy = src(dy, idx);
  m.scale = scale;
  m.W2t = p.w2t; m.W1t = p.w1t;
  m.z1 = z1; m.ld_z1 = 128; m.dx = dx; m.ld_dx = 128;
  return m;
}
static void ffn_bwd(Run& R, const mb_ffn& p, int64_t rows, const float* dy, const int32_t* idx, float scale, const float* z1,
                    float* dx) {
  if (rows == 0) return;
  Scope sc(R);
  mb_mlp_bwd m = ffn_grad(p, rows, dy, idx, scale, z1, dx);
  if (R.scratch) { m.dz1 = R.ar.bottom(rows * 128); m.ld_dz1 = 128; }
  R.op("mb_mlp_bwd_data", [&] { return mb_mlp_bwd_data(&m, R.st); }, 4.0 * rows * 128 * 128, 4.0 * rows * 128 * 3, rows, 128,
       128, 1);
}

// ------------------------------------------------------------------ attention layer
struct AttnInter { float *z1, *z2, *h, *logits, *agg_t, *agg_s, *stats, *z1n, *z2n; };

// keep: the internals go to the top stack and stay; otherwise they are temporaries of the caller's scope (needed: the
// backward pass follows at once) or of this call (nothing will read them again: z1 / z2 are then not written at all).
enum Internals { NONE, TEMP, KEEP };
static void attn_fwd(Run& R, const mb_attn_params& p, const mb_row_graph& g, const float* node, const float* edge,
                     float* node_out, float* edge_out, Internals mode, AttnInter& it) {
  auto get = [&](size_t n) { return mode == KEEP ? R.ar.top(n) : R.ar.bottom(n); };
  const size_t rows = (size_t)g.n_rows, nodes = (size_t)g.n_nodes, ne = (size_t)g.n_edge_rows;
  it.z1 = mode == NONE ? nullptr : get(rows * update_width(p.edge));
  it.z2 = mode == NONE ? nullptr : get(rows * update_width(p.edge));
  it.h = get(rows * 128);
  it.logits = get(ne * 256);
  it.agg_t = get(nodes * 128);
  it.agg_s = get(nodes * 128);
  it.stats = get(nodes * 512);
  it.z1n = mode == NONE ? nullptr : get(nodes * update_width(p.node));
  it.z2n = mode == NONE ? nullptr : get(nodes * update_width(p.node));
  edge_update_fwd(R, p.edge, g, node, edge, nullptr, &p.wst, it.logits, it.z1, it.z2, it.h, p.we, g.is_atom ? nullptr : edge_out);
  R.join(0);  // the logits
  if (g.is_atom && edge_out)
    R.side(0, [&] { MB_OP(mb_pair_mean_res, (int32_t)g.n_edge_rows, g.u2d, g.rev, it.h, edge, p.we, edge_out); });
  MB_OP(mb_seg_attn_fwd, (int32_t)g.n_nodes, g.tgt_ptr, g.src_ptr, g.src_perm, g.emap, it.logits, it.h, it.agg_t, it.agg_s,
        it.stats);
  Scope sc(R);
  float* out = node_out ? node_out : R.ar.bottom(nodes * 128);  // a recomputation wants the internals only
  update_fwd(R, p.node, g.n_nodes, {src(node), src(it.agg_t), src(it.agg_s)}, it.z1n, it.z2n, nullptr, node, p.wn, out);
  R.join(0);
}

static void attn_bwd(Run& R, const mb_attn_params& p, const mb_row_graph& g, const AttnInter& it, const float* d_node_out,
                     const float* d_edge_out, float* d_node, float* d_edge) {
  Scope sc(R);
  const size_t rows = (size_t)g.n_rows, nodes = (size_t)g.n_nodes;
  // node update
  float* dagg_t = R.ar.bottom(nodes * 128);
  float* dagg_s = R.ar.bottom(nodes * 128);
  update_bwd(R, p.node, g.n_nodes, it.z1n, it.z2n, d_node_out, nullptr,
             {{d_node, nullptr, MB_OUT_STORE, d_node_out, p.wn}, {dagg_t, nullptr, MB_OUT_STORE, nullptr, nullptr},
              {dagg_s, nullptr, MB_OUT_STORE, nullptr, nullptr}});
  // softmax-weighted aggregation; dh goes straight on through the gated MLP's tail adjoint (dz2 instead)
  const bool gated = p.edge.kind == MB_UPDATE_GATED;
  float* dz2 = gated ? R.ar.bottom(rows * 256) : nullptr;
  float* dh = gated ? nullptr : R.ar.bottom(rows * 128);
  float* dlogits = R.ar.bottom(rows * 256);
  RowGrad rg{};
  rg.kind = 1; rg.idx_stride = 1;
  rg.dh_in = d_edge_out; rg.dh_map = g.emap; rg.dh_scale = g.is_atom ? 0.5f : 1.f;
  rg.tgt = g.tgt; rg.src = g.src; rg.emap = g.emap;
  rg.logits = it.logits; rg.h = it.h; rg.agg_t = it.agg_t; rg.agg_s = it.agg_s; rg.stats = it.stats; rg.dagg_t = dagg_t;
  rg.dagg_s = dagg_s; rg.dlogits = dlogits; rg.z2 = it.z2; rg.norm_core = p.edge.nc; rg.norm_gate = p.edge.ng;
  if (!gated)
    MB_OP(mb_seg_attn_bwd, g.n_rows, g.tgt, g.src, 1, g.emap, it.logits, it.h, it.agg_t, it.agg_s, it.stats, dagg_t, dagg_s,
          d_edge_out, g.emap, rg.dh_scale, dh, dlogits, nullptr, nullptr, nullptr, nullptr);
  if (gated) {
    edge_update_bwd(R, p.edge, g, it.z1, rg, dz2, g.is_atom ? &p.welt : &p.wstt, d_edge_out, p.we, d_edge, nullptr,
                    nullptr, d_node, nullptr);
    return;
  }
  // edge update (line graph: rows map one to one, so the residual gradient we * d_edge_out rides in the epilogue of the
  // store; atom graph: two directed rows add into one bond row, so it is laid down first)
  const Dest to_tgt{d_node, g.tgt, MB_OUT_ATOMIC, nullptr, nullptr}, to_src{d_node, g.src, MB_OUT_ATOMIC, nullptr, nullptr};
  if (g.is_atom) {
    MB_OP(mb_scale_rows, g.n_edge_rows, d_edge_out, p.we, d_edge, 0);
    update_bwd(R, p.edge, g.n_rows, it.z1, it.z2, dh, dz2, {{d_edge, g.emap, MB_OUT_ATOMIC, nullptr, nullptr}, to_tgt, to_src});
  } else {
    update_bwd(R, p.edge, g.n_rows, it.z1, it.z2, dh, dz2, {{d_edge, nullptr, MB_OUT_STORE, d_edge_out, p.we}, to_tgt, to_src});
  }
  Gemm l(g.n_rows);
  l.block({src(dlogits, nullptr, 0, 256), src(dlogits, nullptr, 128, 256)}, p.wstt, 0, d_edge, 128, 0, g.emap,
          g.is_atom ? MB_OUT_ATOMIC : MB_OUT_ADD);
  l.run(R);
}

// ------------------------------------------------------------------ refinement layer
// Two lines for launches of few bonds, whatever the device (the memory plan depends on them).
// Up to FEW_ENVELOPES bonds the envelopes of all layers come from one launch at the start (42 MB for ten layers at the most).  An
// evaluation with / without it, ms: 156 bonds 2.64 / 2.66, 323 bonds 2.53 / 2.56; 470 - 4,200 bonds between 0.5 % slower and 0.8 % faster;
// 4,400 bonds 5.36 / 5.32, 6,000 bonds 9.81 / 9.68, 7,100 bonds 7.23 / 7.14, 7,600 bonds 8.51 / 8.45 (the side stream that forms an
// envelope beside the layer's products costs nothing there, and its rows are still in L2 when they are read).
constexpr int64_t FEW_ENVELOPES = 4096;
// Up to FEW_BONDS bonds an envelope's gradient goes on into the radial basis's in the kernel that forms it: 1,248 bonds 4.14 -> 4.03 ms,
// 2,300 bonds 4.21 -> 4.10, 4,800 bonds 6.45 -> 6.39, 7,800 bonds 7.72 -> 7.62, 8,200 bonds 7.69 -> 7.64; 11,200 bonds 9.50 and 9.49, 15,200 bonds
// 12.21 -> 12.28, 20,300 bonds 15.61 -> 15.78, where the two separate kernels fill the device.
constexpr int64_t FEW_BONDS = 8192;

struct RefineInter { float *z1, *z2, *h, *env, *zn, *ze; };

static void refine_fwd(Run& R, const mb_refine_params& p, const mb_row_graph& g, int64_t n_bonds, const float* node,
                       const float* edge, const float* rbf, const float* atom_feat, float* node_out, float* edge_out,
                       bool want_edge, Internals mode, RefineInter& it, float* env = nullptr) {
  auto get = [&](size_t n) { return mode == KEEP ? R.ar.top(n) : R.ar.bottom(n); };
  const size_t rows = (size_t)g.n_rows, nodes = (size_t)g.n_nodes;
  it.z1 = mode == NONE ? nullptr : get(rows * update_width(p.edge));
  it.z2 = mode == NONE ? nullptr : get(rows * update_width(p.edge));
  it.h = get(rows * 128);
  it.env = env ? env : get((size_t)n_bonds * 128);
  it.zn = mode == NONE ? nullptr : get(nodes * 128);
  it.ze = mode == NONE || !want_edge ? nullptr : get(rows * 128);
  if (!env) R.side(1, [&] { MB_OP(mb_small_linear_fwd, n_bonds, 7, rbf, p.wenv, it.env); });
  edge_update_fwd(R, p.edge, g, node, edge, g.is_atom ? nullptr : atom_feat, nullptr, nullptr, it.z1, it.z2, it.h, nullptr,
                  nullptr);
  Scope sc(R);
  float* agg = R.ar.bottom(nodes * 128);
  auto node_update = [&] {
    MB_OP(mb_seg_smooth_sum_fwd, (int32_t)g.n_nodes, g.tgt_ptr, g.emap, g.is_atom ? nullptr : g.src, 1, it.env, it.h, agg);
    ffn_fwd(R, p.nffn, g.n_nodes, agg, it.zn, nullptr, node, p.wn, node_out ? node_out : R.ar.bottom(nodes * 128));
  };
  R.join(1);
  if (!want_edge) {  // the last layer's edge update feeds nothing
    node_update();
    return;
  }
  // the edge update reads the unsmoothed rows unless use_smoothed_for_delta_edge (atom graph only,
  // matris/model/interaction_block.py:262-266): then h * s, s = the envelope row of the edge's bond
  const float* x = it.h;
  if (p.smoothed_edge) {
    float* t = R.ar.bottom(rows * 128);
    MB_OP(mb_mul_rows_gather, g.n_rows, it.h, it.env, g.emap, t);
    x = t;
  }
  float* y = g.is_atom || !edge_out ? R.ar.bottom(rows * 128) : nullptr;
  R.side(0, [&] {
    if (g.is_atom) {
      ffn_fwd(R, p.effn, g.n_rows, x, it.ze, y, nullptr, nullptr, nullptr);
      if (edge_out) MB_OP(mb_pair_mean_res, (int32_t)g.n_edge_rows, g.u2d, g.rev, y, edge, p.we, edge_out);
    } else {
      ffn_fwd(R, p.effn, g.n_rows, x, it.ze, nullptr, edge, p.we, edge_out ? edge_out : y);
    }
  });
  node_update();
  R.join(0);
}

static void refine_bwd(Run& R, const mb_refine_params& p, const mb_row_graph& g, int64_t n_bonds, const RefineInter& it,
                       const float* d_node_out, const float* d_edge_out, float* d_node, float* d_edge, float* d_rbf,
                       float* d_atom) {
  Scope sc(R);
  const size_t rows = (size_t)g.n_rows, nodes = (size_t)g.n_nodes;
  const bool want_edge = d_edge_out != nullptr, gated = p.edge.kind == MB_UPDATE_GATED;
  // node FFN
  float* dagg = R.ar.bottom(nodes * 128);
  auto node_ffn = [&] { ffn_bwd(R, p.nffn, g.n_nodes, d_node_out, nullptr, 1.f, it.zn, dagg); };
  // edge FFN
  float* dh = R.ar.bottom(rows * 128);
  const float* drow = nullptr;
  if (want_edge) {
    float* dx = p.smoothed_edge ? R.ar.bottom(rows * 128) : dh;
    const int32_t* const idx = g.is_atom ? g.emap : nullptr;  // (atom graph: the mean over the two directions is a gather * 0.5)
    const float scale = g.is_atom ? 0.5f : 1.f;
    if (R.go() && nodes > 0 && rows > 0 && few_ffn_bwd_fits(g.n_nodes, g.n_rows)) {
      const mb_mlp_bwd a = ffn_grad(p.nffn, g.n_nodes, d_node_out, nullptr, 1.f, it.zn, dagg);
      const mb_mlp_bwd b = ffn_grad(p.effn, g.n_rows, d_edge_out, idx, scale, it.ze, dx);
      const mb_mlp_bwd* const both[2] = {&a, &b};
      R.op("mb_mlp_bwd_data", [&] { return few_ffn_bwd(both, R.st); }, 4.0 * (rows + nodes) * 128 * 128, 4.0 * (rows + nodes) * 128 * 3,
           g.n_rows, 128, 128, 1);
    } else {
      R.side(0, node_ffn);
      ffn_bwd(R, p.effn, g.n_rows, d_edge_out, idx, scale, it.ze, dx);
    }
    if (p.smoothed_edge) {  // dx is the gradient of the smoothed rows h * s
      drow = dx;
      MB_OP(mb_mul_rows_gather, g.n_rows, dx, it.env, g.emap, dh);
    }
    R.join(0);
  } else {
    node_ffn();
  }
  // smoothed aggregation; with a gated update dh is finished in registers and leaves as dz2
  const int32_t* src_idx = g.is_atom ? nullptr : g.src;
  float* dz2 = gated ? R.ar.bottom(rows * 256) : nullptr;
  const bool straight = n_bonds <= FEW_BONDS;  // to the radial basis's gradient
  float* const denv = straight ? nullptr : R.ar.bottom((size_t)n_bonds * 128);
  R.side(1, [&] {
    if (straight) {
      R.op("mb_seg_smooth_sum_bwd_env", [&] {
        return smooth_env_bwd_rbf((int32_t)n_bonds, g, it.env, it.h, dagg, drow, p.wenv, d_rbf, R.st);
      });
      return;
    }
    MB_OP(mb_seg_smooth_sum_bwd_env, (int32_t)n_bonds, g.tgt_ptr, g.is_atom ? nullptr : g.src_ptr, g.src_perm, g.tgt, g.src, 1,
          g.u2d, g.rev, it.env, it.h, dagg, drow, denv);
    MB_OP(mb_small_linear_bwd, n_bonds, 7, denv, p.wenv, d_rbf, 1);
  });
  // edge update
  if (gated) {
    RowGrad rg{};
    rg.kind = 2; rg.idx_stride = 1;
    rg.dh_in = want_edge ? dh : nullptr; rg.tgt = g.tgt; rg.src = src_idx; rg.emap = g.emap; rg.env = it.env; rg.dagg = dagg;
    rg.z2 = it.z2; rg.norm_core = p.edge.nc; rg.norm_gate = p.edge.ng;
    edge_update_bwd(R, p.edge, g, it.z1, rg, dz2, nullptr, d_edge_out, p.we, d_edge, d_node_out, p.wn, d_node, d_atom);
    R.join(1);
    return;
  }
  MB_OP(mb_seg_smooth_sum_bwd_rows, g.n_rows, g.tgt, src_idx, 1, g.emap, it.env, dagg, dh, want_edge ? 1 : 0, nullptr, nullptr, nullptr,
        nullptr);
  R.join(1);
  MB_OP(mb_scale_rows, g.n_nodes, d_node_out, p.wn, d_node, 0);
  const Dest to_tgt{d_node, g.tgt, MB_OUT_ATOMIC, nullptr, nullptr}, to_src{d_node, g.src, MB_OUT_ATOMIC, nullptr, nullptr};
  if (g.is_atom) {
    if (want_edge) MB_OP(mb_scale_rows, g.n_edge_rows, d_edge_out, p.we, d_edge, 0);
    else R.zero(d_edge, (size_t)g.n_edge_rows * 512);
    update_bwd(R, p.edge, g.n_rows, it.z1, it.z2, dh, dz2, {{d_edge, g.emap, MB_OUT_ATOMIC, nullptr, nullptr}, to_tgt, to_src});
  } else {
    update_bwd(R, p.edge, g.n_rows, it.z1, it.z2, dh, dz2,
               {{d_edge, nullptr, MB_OUT_STORE, want_edge ? d_edge_out : nullptr, want_edge ? p.we : nullptr},
                {d_atom, g.ctr, MB_OUT_ATOMIC, nullptr, nullptr}, to_tgt, to_src});
  }
}

// ------------------------------------------------------------------ whole evaluation
static int evaluate(Run& R, mb_eval& E) {
  const mb_model_params& M = *E.model;
  const size_t N = (size_t)E.n_atoms, Ed = (size_t)E.n_edges, Eu = (size_t)E.n_bonds, T = (size_t)E.n_triplets;
  const bool grad = E.f || E.s, line = T > 0;
  const int L = M.n_layers, first_kept = L - (E.keep_layers < L ? E.keep_layers : L);
  Arena& A = R.ar;

  mb_row_graph ga{}, gl{};
  ga.n_rows = E.n_edges; ga.n_nodes = E.n_atoms; ga.n_edge_rows = E.n_bonds; ga.is_atom = 1;
  ga.tgt = E.center; ga.src = E.neighbor; ga.tgt_ptr = E.edge_ptr; ga.src_ptr = E.edge_ptr; ga.src_perm = E.rev;
  ga.emap = E.d2u; ga.u2d = E.u2d; ga.rev = E.rev;
  gl.n_rows = gl.n_edge_rows = E.n_triplets; gl.n_nodes = E.n_bonds; gl.n_ctr = E.n_atoms;
  if (line) {
    gl.ctr = E.lg_cols; gl.tgt = E.lg_cols + T; gl.src = E.lg_cols + 3 * T;
    gl.tgt_ptr = E.trip_ptr; gl.src_ptr = E.trip_src_ptr; gl.src_perm = E.trip_src_perm;
  }

  // gradient buffers of the backward pass, two of each kind (a sub-block reads one and writes the other)
  float *dN[2] = {}, *dE[2] = {}, *dT[2] = {}, *d_rbf2 = nullptr, *d_rbf3 = nullptr;
  if (grad) {
    for (int i = 0; i < 2; ++i) { dN[i] = A.bottom(N * 128); dE[i] = A.bottom(Eu * 128); }
    if (line) for (int i = 0; i < 2; ++i) dT[i] = A.bottom(T * 128);
    d_rbf2 = A.bottom(Eu * 7);
    d_rbf3 = A.bottom(Eu * 7);
  }

  // ---- geometry and embeddings
  float* vec = A.bottom(Ed * 3);
  float* len = A.bottom(Ed);
  float* unit = A.bottom(Ed * 3);
  float* rbf2 = A.bottom(Eu * 7);
  float* rbf3 = A.bottom(Eu * 7);
  MB_OP(mb_edge_geometry_fwd, E.n_edges, E.cart, E.lattice, E.atom_struct, E.center, E.neighbor, E.image, vec, len, unit);
  const int32_t nb = (int32_t)Eu;
  if (M.gaussian) MB_OP(mb_gaussian_fwd, nb, E.u2d, len, M.freq2, M.coeff2, M.freq3, M.coeff3, rbf2, rbf3);
  else MB_OP(mb_bessel_fwd, nb, E.u2d, len, M.freq2, M.cut2, M.freq3, M.cut3, M.envelope_exponent, rbf2, rbf3);

  struct Feat { const float *node, *edge, *trip; };
  std::vector<size_t> low_mark(L);
  std::vector<std::array<size_t, 4>> high_mark(L);  // before line attention, atom attention, line and atom refinement
  std::vector<Feat> in(L + 1), mid(L), half(L);  // layer inputs; after the attentions; after the line refinement
  float* node = A.bottom(N * 128);
  float* edge = A.bottom(Eu * 128);
  float* trip = line ? A.bottom(T * 128) : nullptr;
  const int n_basis = M.fourier ? 7 : 16;
  auto angle_embed = [&](float* basis, float* t1, float* z, int act) {  // z = (act: SiLU of) the triplet embedding's pre-activation
    if (M.fourier) MB_OP(mb_fourier_basis_fwd, E.n_triplets, E.line_graph, unit, M.t_freq, basis);
    else MB_OP(mb_angle_basis_fwd, E.n_triplets, E.line_graph, unit, M.sph_factor, M.cut2, basis);
    MB_OP(mb_small_linear_fwd, E.n_triplets, n_basis, basis, M.t_wa, t1);
    LinearOpt o;
    o.out_act = act;
    linear(R, E.n_triplets, t1, M.t_wb, 128, 128, z, o);
  };
  Scope embed(R);
  if (line) {
    float* basis = A.bottom(T * n_basis);
    float* t1 = A.bottom(T * 128);
    R.side(0, [&] { angle_embed(basis, t1, trip, 1); });
  }
  {
    Scope sc(R);
    float* t = A.bottom(N * 128);
    MB_OP(mb_embedding, E.n_atoms, E.numbers, -1, M.emb_table, t);
    LinearOpt o;
    o.out_act = 1;
    linear(R, E.n_atoms, t, M.emb_w, 128, 128, node, o);
  }
  // bond embedding up to its last layer's input: both directed copies of a bond carry the same row, so the reference's
  // expand-to-directed / average-back pair (matris/model/feature_embed.py:114-148) is the identity here
  auto bond_embed = [&](float* e2, float* e3) {
    Scope sc(R);
    float* e1 = A.bottom(Eu * 128);
    MB_OP(mb_small_linear_fwd, E.n_bonds, 7, rbf2, M.e_w1, e1);
    linear(R, E.n_bonds, e1, M.e_w2, 128, 128, e2);
    MB_OP(mb_layernorm_fwd, E.n_bonds, e2, M.e_lnw, M.e_lnb, e3);
  };
  {
    Scope sc(R);
    float* e2 = A.bottom(Eu * 128);
    float* e3 = A.bottom(Eu * 128);
    bond_embed(e2, e3);
    LinearOpt o;
    o.out_act = 1;
    linear(R, E.n_bonds, e3, M.e_w3, 128, 128, edge, o);
  }
  R.join(0);
  embed.close();

  // ---- interaction blocks.  Without a backward pass the features of a layer live in two sets of buffers used in turn.
  std::vector<AttnInter> ia(L), il(L);
  std::vector<RefineInter> ra(L), rl(L);
  float* ring[2][7] = {};
  if (!grad)
    for (auto& r : ring) {
      for (int i = 0; i < 2; ++i) r[i] = A.bottom(N * 128);
      for (int i = 2; i < 5; ++i) r[i] = A.bottom(Eu * 128);
      if (line) for (int i = 5; i < 7; ++i) r[i] = A.bottom(T * 128);
    }
  std::vector<float*> envs(2 * (size_t)L, nullptr);  // line, atom refinement of each layer
  if (E.n_bonds <= FEW_ENVELOPES && 2 * L <= MANY_LINEARS) {
    ManyLinears many{};
    int n = 0;
    for (int i = 0; i < L; ++i)
      for (int k = line ? 0 : 1; k < 2; ++k, ++n) {
        many.y[n] = envs[2 * i + k] = A.bottom(Eu * 128);
        many.x[n] = k == 0 ? rbf3 : rbf2;
        many.w[n] = k == 0 ? M.layers[i].refine_line.wenv : M.layers[i].refine_atom.wenv;
      }
    R.op("mb_small_linear_fwd", [&] { return many_small_linears(E.n_bonds, n, many, R.st); });
  }
  for (int i = 0; i < L; ++i) {
    const mb_layer_params& P = M.layers[i];
    const Internals mode = !grad ? NONE : (i >= first_kept ? KEEP : NONE);
    const bool last = i == L - 1;
    in[i] = {node, edge, trip};
    low_mark[i] = A.low.size();
    high_mark[i][0] = A.high.size();
    float** r = ring[i & 1];
    float* n_att = grad ? A.bottom(N * 128) : r[0];
    float* n_new = grad ? A.bottom(N * 128) : r[1];
    float* e_att = grad ? A.bottom(Eu * 128) : r[2];
    float* e_at2 = edge;  // without a line graph the edge attention reads the layer's input and its edge output is unused
    float *t_att = nullptr, *t_new = nullptr, *e_ref = edge, *e_new = nullptr;
    if (line) {
      t_att = grad ? A.bottom(T * 128) : r[5];
      if (!last) t_new = grad ? A.bottom(T * 128) : r[6];
      e_at2 = grad ? A.bottom(Eu * 128) : r[3];
      e_ref = grad ? A.bottom(Eu * 128) : r[4];
    }
    if (!last) e_new = grad ? A.bottom(Eu * 128) : (line ? e_at2 : r[3]);
    const float* e_in = edge;
    if (line) {
      Scope sc(R);
      attn_fwd(R, P.attn_line, gl, edge, trip, e_att, t_att, mode, il[i]);
      e_in = e_att;
    }
    high_mark[i][1] = A.high.size();
    {
      Scope sc(R);
      attn_fwd(R, P.attn_atom, ga, node, e_in, n_att, line ? e_at2 : nullptr, mode, ia[i]);
    }
    mid[i] = {n_att, line ? e_at2 : edge, t_att};
    half[i] = {n_att, e_ref, nullptr};
    high_mark[i][2] = A.high.size();
    if (line) {
      Scope sc(R);
      refine_fwd(R, P.refine_line, gl, E.n_bonds, e_at2, t_att, rbf3, n_att, e_ref, t_new, !last, mode, rl[i], envs[2 * i]);
    }
    high_mark[i][3] = A.high.size();
    {
      Scope sc(R);
      // (without gradients e_new may share e_at2's buffer: the line refinement has read it by now)
      refine_fwd(R, P.refine_atom, ga, E.n_bonds, n_att, e_ref, rbf2, nullptr, n_new, e_new, !last, mode, ra[i],
                 envs[2 * i + 1]);
    }
    if (line) half[i].trip = e_att;
    node = n_new;
    if (!last) { edge = e_new; trip = t_new; }
  }

  // ---- heads
  {
    Scope sc(R);
    float* nn = A.bottom(N * 128);
    float* z1 = A.bottom(N * 128);
    float* z2 = A.bottom(N * 128);
    float* ea = A.bottom(N);
    MB_OP(mb_rmsnorm_fwd, E.n_atoms, node, M.out_norm, nn);
    LinearOpt o;
    o.bias = M.h_b0;
    linear(R, E.n_atoms, nn, M.h_w0, 128, 128, z1, o);
    o.bias = M.h_b3; o.in_act = 1;
    linear(R, E.n_atoms, z1, M.h_w3, 128, 128, z2, o);
    MB_OP(mb_head_dot_fwd, E.n_atoms, 128, z2, M.h_w6, M.h_b6, 0, ea);
    R.op("energy_finish", [&] {
      launch(k_energy_finish, cdiv(E.n_struct, FIN_WARPS), 32 * FIN_WARPS, 0, R.st, E.n_struct, E.atom_ptr, ea, E.numbers, M.ref_table, M.n_species, M.is_intensive, E.e, E.ref, E.atoms_per_struct);
      MB_LAUNCH_CHECK("k_energy_finish");
      return (int)MB_OK;
    });
    if (E.m) {
      float* zm = A.bottom(N * 256);
      LinearOpt om;
      om.bias = M.m_b0;
      linear(R, E.n_atoms, nn, M.m_w0, 256, 128, zm, om);
      MB_OP(mb_head_dot_fwd, E.n_atoms, 256, zm, M.m_w3, M.m_b3, 1, E.m);
    }
    if (grad) {
      float* dz2 = A.bottom(N * 128);
      float* dz1 = A.bottom(N * 128);
      MB_OP(mb_head_dot_bwd, E.n_atoms, 128, z2, M.h_w6, nullptr, nullptr, dz2);
      LinearOpt og;
      og.gate = z1;
      linear(R, E.n_atoms, dz2, M.h_w3t, 128, 128, dz1, og);
      linear(R, E.n_atoms, dz1, M.h_w0t, 128, 128, dz2);
      MB_OP(mb_rmsnorm_bwd, E.n_atoms, node, M.out_norm, dz2, dN[0]);
    }
  }
  if (!grad) return R.rc;

  // ---- backward
  R.zero(d_rbf2, Eu * 28);
  R.zero(d_rbf3, Eu * 28);
  bool have_edge = false;  // the last layer's edge outputs carry no gradient
  for (int i = L - 1; i >= 0; --i) {
    const mb_layer_params& P = M.layers[i];
    const bool kept = i >= first_kept, last = i == L - 1;
    const float *n_att = mid[i].node, *e_at2 = mid[i].edge, *t_att = mid[i].trip, *e_ref = half[i].edge, *e_att = half[i].trip;
    auto pop = [&](int which) { A.drop(A.high, A.hi, high_mark[i][which]); };
    // atom refinement: (dN0, dE0) -> (dN1, dE1)
    {
      Scope sc(R);
      if (!kept)
        refine_fwd(R, P.refine_atom, ga, E.n_bonds, n_att, e_ref, rbf2, nullptr, nullptr, nullptr, !last, TEMP, ra[i],
                   envs[2 * i + 1]);
      refine_bwd(R, P.refine_atom, ga, E.n_bonds, ra[i], dN[0], have_edge ? dE[0] : nullptr, dN[1], dE[1], d_rbf2, nullptr);
      pop(3);
    }
    if (line) {
      // line refinement: (dE1, dT0) -> (dE0, dT1), its atom gradient joins dN1
      {
        Scope sc(R);
        if (!kept)
          refine_fwd(R, P.refine_line, gl, E.n_bonds, e_at2, t_att, rbf3, n_att, nullptr, nullptr, !last, TEMP, rl[i],
                     envs[2 * i]);
        refine_bwd(R, P.refine_line, gl, E.n_bonds, rl[i], dE[1], have_edge ? dT[0] : nullptr, dE[0], dT[1], d_rbf3, dN[1]);
        pop(2);
      }
      // atom attention: (dN1, dE0) -> (dN0, dE1)
      {
        Scope sc(R);
        if (!kept) attn_fwd(R, P.attn_atom, ga, in[i].node, e_att, nullptr, nullptr, TEMP, ia[i]);
        attn_bwd(R, P.attn_atom, ga, ia[i], dN[1], dE[0], dN[0], dE[1]);
        pop(1);
      }
      // line attention: (dE1, dT1) -> (dE0, dT0)
      {
        Scope sc(R);
        if (!kept) attn_fwd(R, P.attn_line, gl, in[i].edge, in[i].trip, nullptr, nullptr, TEMP, il[i]);
        attn_bwd(R, P.attn_line, gl, il[i], dE[1], dT[1], dE[0], dT[0]);
        pop(0);
      }
    } else {
      // atom attention, its edge output unused: (dN1, 0) -> (dN0, dE0), then the refinement's edge gradient joins
      Scope sc(R);
      float* none = A.bottom(Eu * 128);
      R.zero(none, Eu * 512);
      if (!kept) attn_fwd(R, P.attn_atom, ga, in[i].node, in[i].edge, nullptr, nullptr, TEMP, ia[i]);
      attn_bwd(R, P.attn_atom, ga, ia[i], dN[1], none, dN[0], dE[0]);
      pop(1);
      MB_OP(mb_scale_rows, E.n_bonds, dE[1], nullptr, dE[0], 1);
    }
    have_edge = true;
    A.drop(A.low, A.lo, low_mark[i]);  // the layer's features have been read for the last time
  }

  // ---- embeddings and geometry, backward
  float* dlen = A.bottom(Ed);
  float* dunit = A.bottom(Ed * 3);
  R.zero(dlen, Ed * 4);
  R.zero(dunit, Ed * 12);
  if (line) {
    float* z = A.bottom(T * 128);
    float* t1 = A.bottom(T * 128);
    float* dz = dT[1];  // free by now
    float* basis = A.bottom(T * n_basis);
    R.side(0, [&] {
      angle_embed(basis, t1, z, 0);
      MB_OP(mb_silu_bwd, E.n_triplets, dT[0], z, dz);
      linear(R, E.n_triplets, dz, M.t_wbt, 128, 128, z);
      MB_OP(mb_small_linear_bwd, E.n_triplets, n_basis, z, M.t_wa, basis, 0);  // its gradient takes the basis's place
      if (M.fourier) MB_OP(mb_fourier_basis_bwd, E.n_triplets, E.line_graph, unit, M.t_freq, basis, dunit);
      else MB_OP(mb_angle_basis_bwd, E.n_triplets, E.line_graph, unit, M.sph_factor, M.cut2, basis, dunit);
    });
  }
  {
    Scope sc(R);
    float* e2 = A.bottom(Eu * 128);
    float* e3 = A.bottom(Eu * 128);
    float* z = A.bottom(Eu * 128);
    float* t = A.bottom(Eu * 128);
    bond_embed(e2, e3);
    linear(R, E.n_bonds, e3, M.e_w3, 128, 128, z);
    MB_OP(mb_silu_bwd, E.n_bonds, dE[0], z, t);
    linear(R, E.n_bonds, t, M.e_w3t, 128, 128, z);
    MB_OP(mb_layernorm_bwd, E.n_bonds, e2, M.e_lnw, z, t);
    linear(R, E.n_bonds, t, M.e_w2t, 128, 128, z);
    MB_OP(mb_small_linear_bwd, E.n_bonds, 7, z, M.e_w1, d_rbf2, 1);
    if (M.gaussian) MB_OP(mb_gaussian_bwd, nb, E.u2d, len, M.freq2, M.coeff2, M.freq3, M.coeff3, d_rbf2, d_rbf3, dlen);
    else MB_OP(mb_bessel_bwd, nb, E.u2d, len, M.freq2, M.cut2, M.freq3, M.cut3, M.envelope_exponent, d_rbf2, d_rbf3, dlen);
  }
  R.join(0);
  float* ge = A.bottom(Ed * 3);
  float* dcart = A.bottom(N * 3);
  float* virial = A.bottom(N * 9);
  float* dstrain = A.bottom((size_t)E.n_struct * 9);
  MB_OP(mb_edge_geometry_bwd, E.n_atoms, E.n_struct, E.n_edges, E.edge_ptr, E.atom_ptr, E.rev, vec, len, unit, dlen, dunit, ge,
        dcart, virial, dstrain);
  R.op("force_stress_finish", [&] {
    const long long n = 3LL * E.n_atoms > 9LL * E.n_struct ? 3LL * E.n_atoms : 9LL * E.n_struct;
    launch(k_force_stress_finish, cdiv(n, 256), 256, 0, R.st, E.n_atoms, E.n_struct, dcart, dstrain, E.volume, E.f, E.s);
    MB_LAUNCH_CHECK("k_force_stress_finish");
    return (int)MB_OK;
  });
  return R.rc;
}

static bool valid(const mb_eval* E) {
  return E && E->model && E->model->layers && E->model->n_layers > 0 && E->n_atoms > 0 && E->n_struct > 0 && E->n_edges > 0 &&
         E->n_bonds > 0 && E->n_triplets >= 0 && E->n_edges < (1LL << 31) && E->n_triplets < (1LL << 31) &&
         E->model->n_species <= FIN_SPECIES;
}

}  // namespace mb

using namespace mb;

// The callers are C: host memory that runs out (the lists of buffers, the layers' bookkeeping) comes back as a status.
template <typename F> static int guarded(F f) {
  try {
    return f();
  } catch (const std::exception&) {
    return MB_ERR_CAPACITY;
  }
}

extern "C" int mb_evaluate_workspace(const mb_eval* e, size_t* bytes) {
  if (!valid(e) || !bytes) return MB_ERR_INVALID;
  return guarded([&] {
    Run R;
    R.scratch = gemm_mode() != 0;
    mb_eval copy = *e;
    const int rc = evaluate(R, copy);
    *bytes = R.ar.peak;
    return rc;
  });
}

extern "C" int mb_evaluate(mb_eval* e, void* stream) {
  if (!valid(e) || (!e->ws && (!e->alloc || !e->release)) || !e->e || !e->cart || !e->numbers || !e->center || (e->n_triplets && (!e->line_graph || !e->lg_cols)))
    return MB_ERR_INVALID;
  Run R;
  R.scratch = gemm_mode() != 0;
  R.st = (cudaStream_t)stream;
  R.ar.mode = e->ws ? Arena::BUFFER : Arena::CALLBACK;
  R.ar.base = (char*)e->ws;
  R.ar.cap = e->ws_bytes;
  R.ar.alloc = e->alloc;
  R.ar.release = e->release;
  Side side;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  // not while every launch is timed by itself, nor with the composed contractions (R.scratch), which drop temporaries on the way
  const bool beside = !R.scratch && !g_times.on && cudaStreamIsCapturing(R.st, &capture) == cudaSuccess &&
                      capture == cudaStreamCaptureStatusNone && side_take(side);
  if (beside) R.sides = &side;
  int rc = guarded([&] { return evaluate(R, *e); });
  if (rc != MB_OK && R.rc == MB_OK) {  // left in the middle of something, perhaps of a branch
    R.rc = rc;
    R.st = (cudaStream_t)stream;
    R.on = 0;
    R.pending[0] = R.pending[1] = beside;
  }
  if (beside) {
    R.join(0);  // (only after an error is anything left)
    R.join(1);
    rc = R.rc;
    if (guarded([&] { side_give(side); return (int)MB_OK; }) != MB_OK) side_free(side);
  }
  e->n_launches = R.launches;
  return rc;
}

static int start_layer(Run& R, void* ws, size_t* ws_bytes, void* stream) {
  if (!ws_bytes) return MB_ERR_INVALID;
  R.scratch = gemm_mode() != 0;
  R.st = (cudaStream_t)stream;
  R.ar.mode = ws ? Arena::BUFFER : Arena::DRY;
  R.ar.base = (char*)ws;
  R.ar.cap = ws ? *ws_bytes : 0;
  return MB_OK;
}

extern "C" int mb_attention_layer(const mb_attn_params* p, const mb_row_graph* g, const float* node, const float* edge,
                                  float* node_out, float* edge_out, const float* d_node_out, const float* d_edge_out,
                                  float* d_node, float* d_edge, void* ws, size_t* ws_bytes, void* stream) {
  Run R;
  if (!p || !g || start_layer(R, ws, ws_bytes, stream)) return MB_ERR_INVALID;
  const bool bwd = d_node_out != nullptr;
  if (ws && (!node || !edge || (bwd && (!d_edge_out || !d_node || !d_edge)))) return MB_ERR_INVALID;
  return guarded([&] {
    AttnInter it;
    attn_fwd(R, *p, *g, node, edge, node_out, edge_out, bwd ? TEMP : NONE, it);
    if (bwd) attn_bwd(R, *p, *g, it, d_node_out, d_edge_out, d_node, d_edge);
    if (!ws) *ws_bytes = R.ar.peak;
    return R.rc;
  });
}

extern "C" int mb_refine_layer(const mb_refine_params* p, const mb_row_graph* g, const float* node, const float* edge,
                               const float* rbf, const float* atom_feat, float* node_out, float* edge_out,
                               const float* d_node_out, const float* d_edge_out, float* d_node, float* d_edge, float* d_rbf,
                               float* d_atom, void* ws, size_t* ws_bytes, void* stream) {
  Run R;
  if (!p || !g || start_layer(R, ws, ws_bytes, stream)) return MB_ERR_INVALID;
  const bool bwd = d_node_out != nullptr, want_edge = bwd ? d_edge_out != nullptr : edge_out != nullptr;
  if (ws && (!node || !edge || !rbf || (bwd && (!d_node || !d_edge || !d_rbf)))) return MB_ERR_INVALID;
  const int64_t n_bonds = g->is_atom ? g->n_edge_rows : g->n_nodes;
  return guarded([&] {
    RefineInter it;
    refine_fwd(R, *p, *g, n_bonds, node, edge, rbf, atom_feat, node_out, edge_out, want_edge, bwd ? TEMP : NONE, it);
    if (bwd) refine_bwd(R, *p, *g, n_bonds, it, d_node_out, d_edge_out, d_node, d_edge, d_rbf, d_atom);
    if (!ws) *ws_bytes = R.ar.peak;
    return R.rc;
  });
}

extern "C" int mb_profile_enable(int on) {
  for (auto& r : g_times.recs) { cudaEventDestroy(r.a); cudaEventDestroy(r.b); }
  g_times.recs.clear();
  g_times.on = on != 0;
  return MB_OK;
}

extern "C" int mb_profile_read(mb_op_record* out, int32_t capacity, int32_t* n) {
  if (!n || (capacity > 0 && !out)) return MB_ERR_INVALID;
  *n = (int32_t)g_times.recs.size();
  if (capacity < *n) return MB_OK;  // called first for the count
  for (int32_t i = 0; i < *n; ++i) {
    OpTimes::Rec& r = g_times.recs[i];
    MB_CUDA_CHECK(cudaEventSynchronize(r.b));
    MB_CUDA_CHECK(cudaEventElapsedTime(&r.r.ms, r.a, r.b));
    out[i] = r.r;
  }
  for (auto& r : g_times.recs) { cudaEventDestroy(r.a); cudaEventDestroy(r.b); }
  g_times.recs.clear();
  return MB_OK;
}
