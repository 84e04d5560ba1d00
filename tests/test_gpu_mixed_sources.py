"""GPU: operands whose 128-wide segments are partly rows in place (by the copy engine) and partly gathered (stored by threads into
the same shared-memory patches), in every order of the two, over several tiles per SM.  Against float64."""
from types import SimpleNamespace

import pytest
import torch
import torch.nn.functional as F

from gpu_util import dev, report

pytestmark = pytest.mark.gpu
TOL = 6e-5  # 3xBF16 operands: 16 mantissa bits per product, sums of a few hundred terms of order one
ROWS = [1, 129, 148 * 128 * 3 + 5]
ORDERS = ["dg", "gd", "dgd", "gdg", "ggd", "gdgd"]  # d: in place, g: gathered


def rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed + sum(shape))
    return (torch.randn(*shape, generator=g) * scale).float()


@pytest.fixture(scope="module")
def ops():
    from matris_b200 import ops as o
    return o


def sources(ops, order, n_rows):
    """(segments for the library, the [n_rows, 128 len(order)] operand they stand for)"""
    x, table = rnd(n_rows, 128 * len(order), seed=1), rnd(61, 128, seed=2)
    g = torch.Generator().manual_seed(n_rows)
    dx, dt, segs, cols = dev(x), dev(table), [], []
    for s, kind in enumerate(order):
        idx = torch.randint(0, 61, (n_rows,), generator=g)
        segs.append(ops.S(dx, None, 128 * s) if kind == "d" else ops.S(dt, dev(idx, torch.int32)))
        cols.append(x[:, 128 * s:128 * s + 128] if kind == "d" else table[idx])
    return segs, torch.cat(cols, 1).double()


@pytest.mark.parametrize("n_rows", ROWS)
@pytest.mark.parametrize("order", ORDERS)
def test_row_gemm(ops, order, n_rows):
    segs, x = sources(ops, order, n_rows)
    W = rnd(256, 128 * len(order), seed=3, scale=0.05)
    dW, out = dev(W), torch.empty(n_rows, 256, device="cuda")
    ops.gemm(n_rows, [ops.B(segs, dW, w_row=128 * j, out=out, out_col=128 * j) for j in (0, 1)])
    assert ops.gemm_status() == 0
    report(f"row GEMM {order} R={n_rows}", out, F.linear(x, W.double()), TOL, scaled=True)
    # column blocks with an operand of their own each, one segment wide
    W1 = rnd(128 * len(order), 128, seed=4, scale=0.09)
    dW1, out = dev(W1), torch.empty(n_rows, 128 * len(order), device="cuda")
    ops.gemm(n_rows, [ops.B([s], dW1, w_row=128 * j, out=out, out_col=128 * j) for j, s in enumerate(segs)])
    assert ops.gemm_status() == 0
    want = torch.cat([F.linear(x[:, 128 * j:128 * j + 128], W1[128 * j:128 * j + 128].double()) for j in range(len(order))], 1)
    report(f"row GEMM, own operands {order} R={n_rows}", out, want, TOL, scaled=True)


@pytest.mark.parametrize("n_rows", ROWS)
@pytest.mark.parametrize("order", ORDERS)
def test_gated_forward_with_residual(ops, order, n_rows):
    segs, x = sources(ops, order, n_rows)
    w1, b1 = rnd(256, 128 * len(order), seed=5, scale=0.05), rnd(256, seed=6)
    w2, b2 = rnd(256, 128, seed=7, scale=0.09), rnd(256, seed=8)
    nc, ng, res, rw = 1 + 0.1 * rnd(128, seed=9), 1 + 0.1 * rnd(128, seed=10), rnd(n_rows, 128, seed=11), rnd(128, seed=12)
    z1 = F.linear(x, w1.double(), b1.double())
    a = F.silu(z1)
    z2 = torch.cat([F.linear(a[:, :128], w2[:128].double()), F.linear(a[:, 128:], w2[128:].double())], 1) + b2.double()
    rms = lambda v, w: v * torch.rsqrt((v * v).mean(1, keepdim=True) + torch.finfo(torch.float32).eps) * w.double()
    h = F.silu(rms(z2[:, :128], nc)) * torch.sigmoid(rms(z2[:, 128:], ng))
    p = SimpleNamespace(w1=dev(w1), b1=dev(b1), w2=dev(w2), b2=dev(b2), nc=dev(nc), ng=dev(ng))
    got = ops.gated_mlp_fwd(p, n_rows, segs, res=dev(res), res_w=dev(rw), save=True)
    assert ops.gemm_status() == 0
    for name, v, w in zip(("z1", "z2", "h", "out2"), got, (z1, z2, h, h + rw.double() * res.double())):
        report(f"gated forward {name} {order} R={n_rows}", v, w, TOL, scaled=True)
