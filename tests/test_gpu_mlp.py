"""GPU: the fused two-layer MLP kernels beyond their plain forward form: gathered addends and the data gradients,
against float64 autograd of the same expressions."""
from types import SimpleNamespace

import pytest
import torch
import torch.nn.functional as F

from gpu_util import dev, report

pytestmark = pytest.mark.gpu
TOL = 6e-5  # 3xBF16 operands: 16 mantissa bits per product, sums of a few hundred terms of order one


def rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).float()


@pytest.fixture(scope="module")
def ops():
    from matris_b200 import ops as o
    return o


def rms(x, w):
    return x * torch.rsqrt((x * x).mean(1, keepdim=True) + torch.finfo(torch.float32).eps) * w


# one row, one ragged tile, a tile edge, one tile per SM and a bit, several tiles per SM (both tile parities)
ROWS = [1, 127, 129, 148 * 128 + 77, 148 * 128 * 2 + 5, 148 * 128 * 5 + 64]


@pytest.mark.parametrize("n_src", [0, 1])
@pytest.mark.parametrize("n_add", [1, 2, 3])
@pytest.mark.parametrize("n_rows", ROWS)
def test_gated_fwd_with_addends(ops, n_rows, n_add, n_src):
    n_nodes = 97
    w1, b1, w2, b2 = rnd(256, 128, scale=0.09), rnd(256, seed=1), rnd(256, 128, seed=2, scale=0.09), rnd(256, seed=3)
    nc, ng = 1 + 0.1 * rnd(128, seed=4), 1 + 0.1 * rnd(128, seed=5)
    x, res, rw = rnd(n_rows, 128, seed=6), rnd(n_rows, 128, seed=7), rnd(128, seed=8)
    g = torch.Generator().manual_seed(n_rows)
    tabs = [rnd(n_nodes, 512, seed=10 + i)[:, 256 * (i % 2):256 * (i % 2) + 256] for i in range(n_add)]
    idx = [torch.randint(0, n_nodes, (n_rows,), generator=g) for _ in range(n_add)]
    z1 = b1.double() + sum(t.double()[i] for t, i in zip(tabs, idx))
    if n_src:
        z1 = z1 + F.linear(x.double(), w1.double())
    a = F.silu(z1)
    z2 = torch.cat([F.linear(a[:, :128], w2[:128].double()), F.linear(a[:, 128:], w2[128:].double())], 1) + b2.double()
    h = F.silu(rms(z2[:, :128], nc.double())) * torch.sigmoid(rms(z2[:, 128:], ng.double()))
    p = SimpleNamespace(w1=dev(w1), b1=dev(b1), w2=dev(w2), b2=dev(b2), nc=dev(nc), ng=dev(ng))
    adds = [(rnd(n_nodes, 512, seed=10 + i).cuda()[:, 256 * (i % 2):256 * (i % 2) + 256], dev(idx[i], torch.int32))
            for i in range(n_add)]
    for save in (True, False):
        got = ops.gated_mlp_fwd(p, n_rows, [ops.S(dev(x))] if n_src else [], res=dev(res), res_w=dev(rw), save=save, adds=adds)
        assert ops.gemm_status() == 0
        want = (z1, z2, h, h + rw.double() * res.double())
        for name, a_, b_ in zip(("z1", "z2", "h", "out2"), got, want):
            if a_ is not None:
                report(f"gated + addends {name} R={n_rows} add={n_add} src={n_src}", a_, b_, TOL, scaled=True)


@pytest.mark.parametrize("n_ext", [0, 1, 2])
@pytest.mark.parametrize("n_rows", ROWS)
def test_gated_bwd(ops, n_rows, n_ext):
    dz2, z1 = rnd(n_rows, 256), rnd(n_rows, 256, seed=1)
    w2t, w1t, w3t = rnd(256, 128, seed=2, scale=0.09), rnd(128, 256, seed=3, scale=0.06), rnd(128, 256, seed=4, scale=0.06)
    ext, res, rw = rnd(n_rows, 256, seed=5), rnd(n_rows, 128, seed=6), rnd(128, seed=7)
    zz = z1.double().requires_grad_(True)
    (sg,) = torch.autograd.grad(F.silu(zz).sum(), zz)
    dz1 = torch.cat([F.linear(dz2[:, :128].double(), w2t[:128].double()), F.linear(dz2[:, 128:].double(), w2t[128:].double())],
                    1) * sg
    dx = F.linear(dz1, w1t.double())
    kw = {}
    if n_ext:
        dx = dx + F.linear(ext[:, :128 * n_ext].double(), w3t[:, :128 * n_ext].double())
        kw = dict(ext=dev(ext)[:, :128 * n_ext], w3t=dev(w3t[:, :128 * n_ext]))
    for with_res in (True, False):
        r = dict(res=dev(res), res_w=dev(rw)) if with_res else {}
        got1, gotx = ops.mlp_bwd(dev(dz2), dev(w2t), dev(w1t), dev(z1), True, **r, **kw)
        assert ops.gemm_status() == 0
        report(f"gated bwd dz1 R={n_rows}", got1, dz1, TOL, scaled=True)
        report(f"gated bwd dx R={n_rows} ext={n_ext}", gotx, dx + (rw.double() * res.double() if with_res else 0), TOL, scaled=True)


@pytest.mark.parametrize("gathered", [False, True])
@pytest.mark.parametrize("n_rows", ROWS)
def test_plain_bwd(ops, n_rows, gathered):
    n_in = 61 if gathered else n_rows
    dy, z1 = rnd(n_in, 128), rnd(n_rows, 128, seed=1)
    idx = torch.randint(0, n_in, (n_rows,), generator=torch.Generator().manual_seed(3)) if gathered else None
    w2t, w1t, res = rnd(128, 128, seed=2, scale=0.09), rnd(128, 128, seed=3, scale=0.09), rnd(n_rows, 128, seed=6)
    zz = z1.double().requires_grad_(True)
    (sg,) = torch.autograd.grad(F.silu(zz).sum(), zz)
    rows = dy.double()[idx] if gathered else dy.double()
    dz1 = 0.5 * F.linear(rows, w2t.double()) * sg
    dx = F.linear(dz1, w1t.double())
    di = dev(idx, torch.int32) if gathered else None
    got1, gotx = ops.mlp_bwd(dev(dy), dev(w2t), dev(w1t), dev(z1), False, idx=di, scale=0.5)
    report(f"plain bwd dz1 R={n_rows}", got1, dz1, TOL, scaled=True)
    report(f"plain bwd dx R={n_rows}", gotx, dx, TOL, scaled=True)
    none, gotx = ops.mlp_bwd(dev(dy), dev(w2t), dev(w1t), dev(z1), False, idx=di, scale=0.5, want_dz1=False, res=dev(res))
    assert none is None and ops.gemm_status() == 0
    report(f"plain bwd dx + res R={n_rows}", gotx, dx + res.double(), TOL, scaled=True)


def test_composed_modes_agree(ops):
    """The other GEMM modes build the same results from separate launches."""
    R, n_nodes = 1000 + 3, 50
    w1, b1, w2, b2 = rnd(256, 128, scale=0.09), rnd(256, seed=1), rnd(256, 128, seed=2, scale=0.09), rnd(256, seed=3)
    p = SimpleNamespace(w1=dev(w1), b1=dev(b1), w2=dev(w2), b2=dev(b2), nc=dev(1 + 0 * rnd(128)), ng=dev(1 + 0 * rnd(128)))
    x, idx = dev(rnd(R, 128, seed=6)), dev(torch.randint(0, n_nodes, (R,), generator=torch.Generator().manual_seed(1)), torch.int32)
    tab, ext, w3t = dev(rnd(n_nodes, 256, seed=9)), dev(rnd(R, 256, seed=5)), dev(rnd(128, 256, seed=4, scale=0.06))
    w1t, res = dev(w1.t().contiguous()), dev(rnd(R, 128, seed=6))
    outs = {}
    try:
        for mode in ("simt", "tcgen05_tile", "tcgen05_tf32", "tcgen05"):
            ops.set_gemm_mode(mode)
            z1, z2, h, _ = ops.gated_mlp_fwd(p, R, [ops.S(x)], adds=[(tab, idx)])
            only = ops.gated_mlp_fwd(p, R, [], adds=[(tab, idx)])[2]
            dz1, dx = ops.mlp_bwd(z2, dev(w2), w1t, z1, True, res=res, ext=ext, w3t=w3t)
            dp, dq = ops.mlp_bwd(x, dev(w2[:128]), dev(w2[128:]), x, False, scale=0.5)
            outs[mode] = (z1, z2, h, only, dz1, dx, dp, dq)
            assert ops.gemm_status() == 0
    finally:
        ops.set_gemm_mode("tcgen05")
    for mode in ("tcgen05_tile", "tcgen05_tf32", "tcgen05"):
        for i, (a, b) in enumerate(zip(outs[mode], outs["simt"])):
            report(f"mode {mode} output {i}", a, b, TOL, scaled=True)
