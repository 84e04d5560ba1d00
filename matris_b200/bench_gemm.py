"""Kernel micro-benchmark: one `mb_gemm`, `mb_gated_mlp_fwd` or `mb_mlp_bwd_data` launch shape, timed with CUDA events (median of
nine launches, each behind a write of twice the L2).

    python -m matris_b200.bench_gemm K N [act] [gate] [rows] [mode] [scatter]
    python -m matris_b200.bench_gemm gated K [rows] [save] [res] [gather] [adds]
    python -m matris_b200.bench_gemm ffn K [rows] [save] [res]
    python -m matris_b200.bench_gemm bwd gated|plain [rows] [res] [ext]

ffn: the plain two-layer form of the fused kernel (K -> 128 -> 128, `ops.ffn_fwd`); save: also write z1 (default 1);
res: write out2 = y + res_w * res instead of y (default 1).
gated: the fused gated-MLP forward (K -> 256 -> 2 x 128 -> 128); save: also write z1 / z2 (default 1); res: also
write out2 = h + res_w * res (default 1); gather: 1 = K segments 1.. are gathered from a table of rows/6 rows through
random indices (default 0: all segments read row r); adds: that many addends gathered from tables of rows/5 rows in sorted
order (K may then be 0).
bwd: the data gradient of a gated (256 -> 128, ext: further 128-wide segments) or plain (128 -> 128) two-layer MLP; res: plus the
residual's gradient (default 1).

K: reduction width (a multiple of 128: K/128 concatenated sources), N: output width (a multiple of 128: N/128 column
blocks), act: SiLU on load, gate: SiLU' gate in the epilogue, rows: default 151,552 (8 tiles per SM on 148 SMs),
mode: tcgen05 (persistent 3xBF16 kernel, default) | tcgen05_tf32 | tcgen05_tile | simt; scatter: 0 plain store (default), 1 atomic
scatter-add to rows/5 targets in sorted order (runs of five equal targets), 2 the same targets in random order.
"""
import sys

import torch

from matris_b200 import ops


def timed(launch):
    """Milliseconds of a launch."""
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    times = []
    for i in range(12):
        flush.fill_(i)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        launch()
        e1.record()
        times.append((e0, e1))
    torch.cuda.synchronize()
    assert ops.gemm_status() == 0
    return sorted(a.elapsed_time(b) for a, b in times[3:])[4]


def gated(argv):
    from types import SimpleNamespace
    K = int(argv[0])
    rows = int(argv[1]) if len(argv) > 1 else 148 * 128 * 8
    save = bool(int(argv[2])) if len(argv) > 2 else True
    with_res = bool(int(argv[3])) if len(argv) > 3 else True
    gather = bool(int(argv[4])) if len(argv) > 4 else False
    n_add = int(argv[5]) if len(argv) > 5 else 0
    torch.manual_seed(0)
    dev = "cuda"
    p = SimpleNamespace(w1=ops.SplitWeight(torch.randn(256, max(K, 128), device=dev) * max(K, 128) ** -0.5), b1=torch.randn(256, device=dev) * 0.1,
                        w2=ops.SplitWeight(torch.randn(256, 128, device=dev) * 128 ** -0.5),
                        b2=torch.randn(256, device=dev) * 0.1, nc=torch.ones(128, device=dev), ng=torch.ones(128, device=dev))
    x = torch.randn(rows, 128, device=dev)
    srcs = [ops.S(x)] if K else []
    sorted_idx = (torch.arange(rows, device=dev) // 5).to(torch.int32)
    adds = [(torch.randn(rows // 5 + 1, 256, device=dev), sorted_idx) for _ in range(n_add)]
    if gather:
        table = torch.randn(rows // 6 + 1, 128, device=dev)
        for s_ in range(K // 128 - 1):
            idx = torch.randint(0, table.shape[0], (rows,), device=dev, dtype=torch.int32)
            srcs.append(ops.S(table, idx))
    else:
        more = torch.randn(rows, K - 128, device=dev) if K > 128 else None
        srcs += [ops.S(more, None, 128 * s_) for s_ in range(K // 128 - 1)]
    res = torch.randn(rows, 128, device=dev) if with_res else None
    rw = torch.randn(128, device=dev) if with_res else None

    ms = timed(lambda: ops.gated_mlp_fwd(p, rows, srcs, want_h=not with_res, res=res, res_w=rw, save=save, adds=adds))
    flops = 2.0 * rows * 256 * (K + 128)
    gbytes = 4.0 * rows * (K + 128 * (1 + 4 * save + with_res)) / 1e9
    print(f"gated rows={rows} K={K} save={int(save)} res={int(with_res)} gather={int(gather)} adds={n_add}: {ms:.3f} ms, "
          f"{flops / ms / 1e9:.1f} TFLOP/s fp32-equivalent, {gbytes / ms * 1e3:.0f} GB/s of algorithmic traffic")


def ffn(argv):
    from types import SimpleNamespace
    K = int(argv[0])
    rows = int(argv[1]) if len(argv) > 1 else 148 * 128 * 8
    save = bool(int(argv[2])) if len(argv) > 2 else True
    with_res = bool(int(argv[3])) if len(argv) > 3 else True
    torch.manual_seed(0)
    dev = "cuda"
    p = SimpleNamespace(w1=ops.SplitWeight(torch.randn(128, K, device=dev) * K ** -0.5), b1=torch.randn(128, device=dev) * 0.1,
                        w2=ops.SplitWeight(torch.randn(128, 128, device=dev) * 128 ** -0.5),
                        b2=torch.randn(128, device=dev) * 0.1)
    x = torch.randn(rows, K, device=dev)
    res = torch.randn(rows, 128, device=dev) if with_res else None
    rw = torch.randn(128, device=dev) if with_res else None

    ms = timed(lambda: ops.ffn_fwd(p, x, want_y=not with_res, res=res, res_w=rw, save=save))
    flops = 2.0 * rows * 128 * (K + 128)
    gbytes = 4.0 * rows * (K + 128 * (1 + save + with_res)) / 1e9
    print(f"ffn rows={rows} K={K} save={int(save)} res={int(with_res)}: {ms:.3f} ms, "
          f"{flops / ms / 1e9:.1f} TFLOP/s fp32-equivalent, {gbytes / ms * 1e3:.0f} GB/s of algorithmic traffic")


def bwd(argv):
    is_gated = argv[0] == "gated"
    rows = int(argv[1]) if len(argv) > 1 else 148 * 128 * 8
    with_res = bool(int(argv[2])) if len(argv) > 2 else True
    n_ext = int(argv[3]) if len(argv) > 3 else 0
    torch.manual_seed(0)
    dev, width = "cuda", 256 if is_gated else 128
    dy, z1 = torch.randn(rows, width, device=dev), torch.randn(rows, width, device=dev)
    w2t, w1t = (ops.SplitWeight(torch.randn(a, b, device=dev) * 0.09) for a, b in ((width, 128), (128, width)))
    kw = {}
    if n_ext:
        kw.update(ext=torch.randn(rows, 128 * n_ext, device=dev), w3t=ops.SplitWeight(torch.randn(128, 128 * n_ext, device=dev) * 0.06))
    if with_res:
        kw.update(res=torch.randn(rows, 128, device=dev), res_w=torch.randn(128, device=dev))
    ms = timed(lambda: ops.mlp_bwd(dy, w2t, w1t, z1, is_gated, want_dz1=is_gated, **kw))
    gbytes = 4.0 * rows * 128 * ((7 if is_gated else 3) + with_res + n_ext) / 1e9
    print(f"bwd {argv[0]} rows={rows} res={int(with_res)} ext={n_ext}: {ms:.3f} ms, {gbytes / ms * 1e3:.0f} GB/s of algorithmic traffic")


def main(argv):
    if argv[0] == "bwd":
        return bwd(argv[1:])
    if argv[0] == "gated":
        return gated(argv[1:])
    if argv[0] == "ffn":
        return ffn(argv[1:])
    K, N = int(argv[0]), int(argv[1])
    act = int(argv[2]) if len(argv) > 2 else 0
    gate = int(argv[3]) if len(argv) > 3 else 0
    rows = int(argv[4]) if len(argv) > 4 else 148 * 128 * 8
    mode = argv[5] if len(argv) > 5 else "tcgen05"
    scatter = int(argv[6]) if len(argv) > 6 else 0
    torch.manual_seed(0)
    x = torch.randn(rows, K, device="cuda")
    z = torch.randn(rows, N, device="cuda") if gate else None
    W = ops.SplitWeight((torch.randn(N, K, device="cuda") * 0.1).contiguous())
    out = torch.empty(rows, N, device="cuda")
    out_idx, out_mode = None, ops.OUT_STORE
    if scatter:
        out_idx = (torch.arange(rows, device="cuda") // 5).to(torch.int32)
        if scatter == 2:
            out_idx = out_idx[torch.randperm(rows, device="cuda")].contiguous()
        out = torch.zeros(rows // 5 + 1, N, device="cuda")
        out_mode = ops.OUT_ATOMIC
    ops.set_gemm_mode(mode)

    def launch():
        ops.gemm(rows, [ops.B([ops.S(x, None, 128 * s, act=act) for s in range(K // 128)], W, w_row=128 * j, out=out,
                              out_col=128 * j, gate=z, gate_col=128 * j if gate else 0, out_idx=out_idx, mode=out_mode)
                        for j in range(N // 128)])

    ms = timed(launch)
    print(f"rows={rows} K={K} N={N} act={act} gate={gate} mode={mode} scatter={scatter}: {ms:.3f} ms, "
          f"{2.0 * rows * K * N / ms / 1e9:.1f} TFLOP/s fp32-equivalent")


if __name__ == "__main__":
    main(sys.argv[1:])
