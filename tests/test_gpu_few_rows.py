"""GPU: the kernel for few rows (csrc/few_rows.cuh) against float64, and bit for bit against the persistent kernels: a row's result
does not depend on how many rows a call has."""
from types import SimpleNamespace

import pytest
import torch
import torch.nn.functional as F

from gpu_util import dev, report
from test_gpu_mlp import TOL, rms, rnd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from matris_b200 import ops as o
    return o


def sizes():
    """One row, edges of the tiles, the last launch of each tile height and the first of the next (the last one: persistent kernels)."""
    n = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 1
    return [1, 15, 17, 33, 16 * n, 16 * n + 1, 32 * n - 1, 32 * n + 1, 64 * n, 64 * n + 1]


BIG = 40_000


@pytest.mark.parametrize("at", range(10))
@pytest.mark.parametrize("k,n,mode", [(128, 128, "plain"), (512, 128, "res"), (128, 512, "gate"), (256, 256, "add")])
def test_dense(ops, k, n, mode, at):
    rows = sizes()[at]
    x, w, b, z, res, rw = rnd(BIG, k), rnd(n, k, seed=1, scale=k ** -0.5), rnd(n, seed=2), rnd(BIG, n, seed=3), rnd(BIG, n, seed=4), rnd(n, seed=5)
    dx, dw, db, dz, dres, drw = dev(x), ops.SplitWeight(dev(w)), dev(b), dev(z), dev(res), dev(rw)
    idx = torch.randperm(BIG, generator=torch.Generator().manual_seed(6))
    di = dev(idx, torch.int32)

    def run(r):
        out = dres[:r].clone() if mode == "add" else torch.full((r, n), 7.0, device="cuda")
        ops.gemm(r, [ops.B([ops.S(dx, di[:r] if mode == "plain" else None, 128 * s, act=int(mode == "gate")) for s in range(k // 128)], dw,
                           w_row=128 * j, out=out, out_col=128 * j, bias=db[128 * j:128 * j + 128], out_act=int(mode == "plain"),
                           gate=dz if mode == "gate" else None, gate_col=128 * j if mode == "gate" else 0,
                           res=dres if mode == "res" else None, res_w=drw[128 * j:128 * j + 128] if mode == "res" else None,
                           res_col=128 * j if mode == "res" else 0, mode=ops.OUT_ADD if mode == "add" else ops.OUT_STORE)
                     for j in range(n // 128)])
        return out

    got = run(rows)
    assert ops.gemm_status() == 0
    a = x.double()[idx[:rows]] if mode == "plain" else x.double()[:rows]
    want = F.linear(F.silu(a) if mode == "gate" else a, w.double(), b.double())
    zz = z[:rows].double().requires_grad_(True)
    (sg,) = torch.autograd.grad(F.silu(zz).sum(), zz)
    want = {"plain": F.silu(want), "res": want + rw.double() * res[:rows].double(), "gate": want * sg,
            "add": want + res[:rows].double()}[mode]
    report(f"few rows {k}->{n} {mode} R={rows}", got, want, TOL, scaled=True)
    assert torch.equal(got, run(BIG)[:rows])


@pytest.mark.parametrize("at", range(10))
def test_mlps(ops, at):
    rows = sizes()[at]
    n_nodes = 61
    w = {s: dev(rnd(*s, seed=i, scale=s[1] ** -0.5)) for i, s in enumerate([(256, 128), (256, 384), (128, 128), (128, 256)])}
    b1, b2, nc, ng, rw = (dev(rnd(m, seed=10 + i)) for i, m in enumerate([256, 256, 128, 128, 128]))
    x, res, z1, ext = (dev(rnd(BIG, m, seed=20 + i)) for i, m in enumerate([384, 128, 256, 256]))
    tab = dev(rnd(n_nodes, 256, seed=30))
    idx = dev(torch.randint(0, n_nodes, (BIG,), generator=torch.Generator().manual_seed(1)), torch.int32)
    p = SimpleNamespace(w1=w[256, 128], b1=b1, w2=w[256, 128], b2=b2, nc=nc, ng=ng)
    wide = SimpleNamespace(w1=w[256, 384], b1=b1, w2=w[256, 128], b2=b2, nc=nc, ng=ng)
    f = SimpleNamespace(w1=w[128, 128], b1=b1[:128], w2=w[128, 128], b2=b2[:128])

    def run(r):
        s = ops.S
        return {
            "gated": ops.gated_mlp_fwd(p, r, [s(x)], res=res[:r], res_w=rw, adds=[(tab, idx[:r]), (tab, idx.flip(0)[:r].contiguous())]),
            "gated, K = 384": ops.gated_mlp_fwd(wide, r, [s(x), s(tab, idx[:r]), s(x, None, 256)]),
            "gated, addends only": ops.gated_mlp_fwd(p, r, [], adds=[(tab, idx[:r])] * 3, save=False),
            "ffn": ops.ffn_fwd(f, x[:r, :128].contiguous(), want_y=True, res=res[:r], res_w=rw),
            "gated backward": ops.mlp_bwd(z1[:r], w[256, 128], w[128, 256], x[:r, :256], True, ext=ext[:r], w3t=w[128, 256], res=res[:r], res_w=rw),
            "ffn backward": ops.mlp_bwd(tab[:, :128].contiguous(), w[128, 128], w[128, 128], res[:r], False, idx=idx[:r], scale=0.5),
        }

    small, big = run(rows), run(BIG)
    assert ops.gemm_status() == 0
    for name, outs in small.items():
        for i, (a, b) in enumerate(zip(outs, big[name])):
            assert (a is None) == (b is None)
            if a is not None:
                assert torch.equal(a, b[:rows]), (name, i)
    # one form against float64 (the others: test_gpu_mlp.py, whose smallest sizes take the same kernel)
    z = F.linear(torch.cat([x[:rows, :128], tab[idx[:rows].long()][:, :128], x[:rows, 256:]], 1).double(), w[256, 384].double(), b1.double())
    a = F.silu(z)
    y = torch.cat([F.linear(a[:, :128], w[256, 128][:128].double()), F.linear(a[:, 128:], w[256, 128][128:].double())], 1) + b2.double()
    h = F.silu(rms(y[:, :128], nc.double())) * torch.sigmoid(rms(y[:, 128:], ng.double()))
    for name, got, want in zip(("z1", "z2", "h"), small["gated, K = 384"], (z, y, h)):
        report(f"few rows gated K=384 {name} R={rows}", got, want, TOL, scaled=True)


@pytest.mark.parametrize("options", [{}, dict(use_bias=True, use_smoothed_for_delta_edge=True)])
def test_small_structures_equal_their_batch(options):
    """Alone, a small structure takes the few-row kernels, merged launches and gradients formed on the way; in a large batch its rows
    take the row kernels and the persistent contractions.  The expressions are the same; sums over atoms' rows may meet in another
    order (rounding of float32 sums of order one)."""
    from matris_b200 import MatRIS, workloads
    from matris_b200.weights import random_checkpoint
    from conftest import GPA
    small = [workloads.cu_fcc((1, 1, 1), sigma=0.05), workloads.demo_pu4si6(), workloads.cu_fcc((2, 2, 2), sigma=0.05),
             workloads.random_crystals(1, seed=3)[0]]
    model = MatRIS.from_dict(random_checkpoint(dict(num_layers=2, reference_energy="mpa", **options), seed=1, jitter=0.1)).to("cuda")
    many = model.predict(small * 40, "efsm")
    for i, c in enumerate(small):
        one = model.predict([c], "efsm")
        report(f"alone vs in a batch {i}: E", one["e"][0], many["e"][i], 1e-6, scaled=True)
        report(f"alone vs in a batch {i}: F", one["f"][0], many["f"][i], 2e-6)
        report(f"alone vs in a batch {i}: S", one["s"][0] / GPA, many["s"][i] / GPA, 2e-7)
        report(f"alone vs in a batch {i}: M", one["m"][0], many["m"][i], 2e-6)


@pytest.mark.parametrize("count", [61, 125])
def test_sums_of_a_bonds_two_rows_as_operand(count):
    """A bond's gradient contracts the sums of its two directed rows.  156 bonds a structure: 75 row tiles, the last of 44 rows, one
    for each column block a multiprocessor; and 153, more than one for some.  Alone, a structure takes the few-row kernel."""
    from matris_b200 import MatRIS, workloads
    from matris_b200.weights import random_checkpoint
    from conftest import GPA
    c = workloads.cu_fcc((1, 1, 1), sigma=0.05)
    model = MatRIS.from_dict(random_checkpoint(dict(num_layers=2, reference_energy="mpa"), seed=1, jitter=0.1)).to("cuda")
    one, many = model.predict([c], "efs"), model.predict([c] * count, "efs")
    for i in range(count):  # tolerances as above: the same expressions, float32 sums of order one in another order
        report(f"bond sums {count}/{i}: F", one["f"][0], many["f"][i], 2e-6)
        report(f"bond sums {count}/{i}: S", one["s"][0] / GPA, many["s"][i] / GPA, 2e-7)
