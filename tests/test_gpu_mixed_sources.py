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


@pytest.mark.parametrize("stride", [0, 64])
@pytest.mark.parametrize("n_rows", [1, 300, 148 * 128 + 77])
def test_rows_that_share_memory(ops, n_rows, stride):
    """Row strides shorter than a row: one row for all (0) and overlapping windows (64), as operand, gate and residual."""
    def rows(seed):
        return rnd(64 * n_rows + 128, seed=seed).cuda().as_strided((n_rows, 128), (stride, 1))
    x, z, r = rows(1), rows(2), rows(3)
    full = [t.cpu().double() for t in (x, z, r)]
    W, rw = rnd(128, 128, seed=4, scale=0.09), rnd(128, seed=5)
    zz = full[1].clone().requires_grad_(True)
    (sg,) = torch.autograd.grad(F.silu(zz).sum(), zz)
    y = ops.linear(x, dev(W), gate=z, res=r, res_w=dev(rw))
    report(f"row GEMM stride {stride} R={n_rows}", y, F.linear(full[0], W.double()) * sg + rw.double() * full[2], TOL, scaled=True)
    w1, w2 = rnd(128, 128, seed=6, scale=0.09), rnd(128, 128, seed=7, scale=0.09)
    p = SimpleNamespace(w1=dev(w1), b1=None, w2=dev(w2), b2=None)
    _, got, out2 = ops.ffn_fwd(p, x, res=r, res_w=dev(rw))
    want = F.linear(F.silu(F.linear(full[0], w1.double())), w2.double())
    report(f"FFN stride {stride} R={n_rows}", got, want, TOL, scaled=True)
    report(f"FFN + residual stride {stride} R={n_rows}", out2, want + rw.double() * full[2], TOL, scaled=True)
    assert ops.gemm_status() == 0
