"""GPU: the kernel for few rows (csrc/few_rows.cuh) against float64, and bit for bit against the persistent kernels: a row's result
does not depend on how many rows a call has."""
from types import SimpleNamespace

import numpy as np
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


# ------------------------------------------------------------------ sub-blocks: merged launches, row gradients, sums of two rows
def grouped(key, n):
    """Row numbers sorted by key (stable) and the start of each key's run."""
    return np.argsort(key, kind="stable"), np.concatenate([[0], np.cumsum(np.bincount(key, minlength=n))])


def line_graph(rows, nodes, seed):
    """Rows sorted by target node; two target nodes share a centre, so that a centre's sum is of two terms at the most."""
    r = np.random.default_rng(seed)
    tgt, src = np.sort(r.integers(0, nodes, rows)), r.integers(0, nodes, rows)
    perm, src_ptr = grouped(src, nodes)
    return dict(n_rows=rows, n_nodes=nodes, n_edge_rows=rows, n_ctr=(nodes + 1) // 2, tgt=tgt, src=src, ctr=tgt // 2, src_perm=perm,
                tgt_ptr=grouped(tgt, nodes)[1], src_ptr=src_ptr)


def atom_graph(bonds, nodes, seed):
    """Two directed rows a bond, sorted by centre."""
    r = np.random.default_rng(seed)
    a, b = r.integers(0, nodes, (2, bonds))
    order, ptr = grouped(np.concatenate([a, b]), nodes)
    at = np.empty(2 * bonds, dtype=np.int64)
    at[order] = np.arange(2 * bonds)  # where a directed row went
    bond, rev = order % bonds, at[(order + bonds) % (2 * bonds)]
    return dict(n_rows=2 * bonds, n_nodes=nodes, n_edge_rows=bonds, n_ctr=0, is_atom=1, tgt=np.concatenate([a, b])[order],
                src=np.concatenate([b, a])[order], tgt_ptr=ptr, src_ptr=ptr, src_perm=rev, rev=rev, emap=bond, u2d=at[:bonds])


def joined(g, h):
    """Both graphs as one, the first's rows, nodes and bonds first."""
    of = dict(tgt="n_nodes", src="n_nodes", ctr="n_ctr", src_perm="n_rows", rev="n_rows", u2d="n_rows", emap="n_edge_rows", tgt_ptr="n_rows",
              src_ptr="n_rows")
    out = {k: g[k] + h[k] for k in ("n_rows", "n_nodes", "n_edge_rows", "n_ctr")}
    out.update({k: np.concatenate([g[k], h[k][int(k.endswith("_ptr")):] + g[of[k]]]) for k in of if k in g})
    return {**out, "is_atom": g.get("is_atom", 0)}


def on_device(g):
    from matris_b200 import _lib
    alive = {k: dev(v, torch.int32) for k, v in g.items() if isinstance(v, np.ndarray)}
    c = _lib.MbRowGraph(**{k: int(v) for k, v in g.items() if not isinstance(v, np.ndarray)}, **{k: _lib.ptr(v) for k, v in alive.items()})
    return SimpleNamespace(c=c, alive=alive, skip_edge_out=False)


@pytest.fixture(scope="module")
def layer():
    from matris_b200.model import pack_parameters
    from matris_b200.weights import full_config, random_checkpoint
    ck = random_checkpoint(dict(num_layers=1), seed=3, jitter=0.1)
    return pack_parameters(ck["state_dict"], full_config(ck["config"]), torch.device("cuda"))


def sub_block(layer, kind, g, x):
    """Results and gradients of a sub-block on the first rows of the features x."""
    from matris_b200.model import AttentionFn, RefineFn
    line = not g.get("is_atom")
    bonds = g["n_nodes"] if line else g["n_edge_rows"]
    node, edge, rbf, atom = (x[k][:n].clone().requires_grad_(True) for k, n in (("node", g["n_nodes"]), ("edge", g["n_edge_rows"]),
                                                                                ("rbf", bonds), ("atom", g["n_ctr"])))
    P, rg = getattr(layer.layers[0], f"{kind}_{'line' if line else 'atom'}"), on_device(g)
    if kind == "attn":
        leaves, out = [node, edge], AttentionFn.apply(node, edge, P, rg)
    else:
        leaves = [node, edge, rbf] + [atom] * line
        out = RefineFn.apply(node, edge, rbf, atom if line else None, P, rg)
    grads = torch.autograd.grad(out, leaves, [x["d_node"][:g["n_nodes"]], x["d_edge"][:g["n_edge_rows"]]])
    return [t.detach() for t in (*out, *grads)]


def compare(layer, ops, kind, small, big, seed):
    both = joined(small, big)
    n = max(both[k] for k in ("n_nodes", "n_edge_rows", "n_ctr"))
    x = {k: dev(rnd(n, w, seed=seed + i)) for i, (k, w) in enumerate([("node", 128), ("edge", 128), ("rbf", 7), ("atom", 128),
                                                                      ("d_node", 128), ("d_edge", 128)])}
    alone, among = sub_block(layer, kind, small, x), sub_block(layer, kind, both, x)
    assert ops.gemm_status() == 0
    for i, (a, b) in enumerate(zip(alone, among)):
        assert torch.isfinite(a).all() and torch.equal(a, b[:a.shape[0]]), (i, (a - b[:a.shape[0]]).abs().max())


def shapes():
    """(rows, nodes) at the edges of the tiles: row gradients with one output take n rows a tile, with three (the node update's) a third."""
    n = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 3
    t = n // 3
    return [(1, 1), (15, 7), (17, 16), (33, 17), (16 * n, 16 * t), (16 * n + 1, 16 * t + 1), (32 * n - 1, 32 * t), (32 * n, 32 * t + 1),
            (32 * n + 1, 16 * n), (64 * n, 16 * n + 1), (64 * n + 1, 32 * n)]


@pytest.mark.parametrize("at", range(11))
@pytest.mark.parametrize("kind", ["attn", "refine"])
@pytest.mark.parametrize("which", ["line", "atom"])
def test_sub_blocks_do_not_depend_on_how_many_rows_there_are(layer, ops, which, kind, at):
    """Alone, a graph's sub-block takes merged launches (of problems with different numbers of rows), row gradients formed inside the
    products and sums of a bond's two rows as operand; in front of a large graph, the row kernels and the persistent contractions.  All
    sums keep their order, so the results of the first graph's rows are the same bit for bit."""
    rows, nodes = shapes()[at]
    if which == "line":
        compare(layer, ops, kind, line_graph(rows, nodes, at), line_graph(50_000, 10_000, 99), 10 * at)
    else:  # segments of 16 rows and more on both sides: the kernel of the sums of node rows is chosen by that
        small = atom_graph((rows + 1) // 2, max(1, rows // 20), at) if rows > 40 else atom_graph((rows + 1) // 2, 1, at)
        compare(layer, ops, kind, small, atom_graph(90_000, 9_600, 99), 10 * at)


@pytest.mark.parametrize("bonds", [8192, 8193])
@pytest.mark.parametrize("which", ["line", "atom"])
def test_envelope_gradient_either_side_of_its_line(layer, ops, which, bonds):
    """Up to 8,192 bonds the envelopes' gradient goes straight on into the radial basis's."""
    if which == "line":
        compare(layer, ops, "refine", line_graph(3 * bonds, bonds, 1), line_graph(6_000, 2_000, 2), 5)
    else:
        compare(layer, ops, "refine", atom_graph(bonds, 700, 1), atom_graph(2_000, 150, 2), 5)


def test_energies_either_side_of_the_line_of_merged_envelopes():
    """156 bonds a structure: 26 of them stay below 4,096 bonds, 27 do not.  No sum of the forward pass depends on the batch."""
    from matris_b200 import MatRIS, workloads
    from matris_b200.weights import random_checkpoint
    c = workloads.cu_fcc((1, 1, 1), sigma=0.05)
    model = MatRIS.from_dict(random_checkpoint(dict(num_layers=2, reference_energy="mpa"), seed=1, jitter=0.1)).to("cuda")
    one = model.predict([c], "efs")
    for count in (26, 27):
        g = model.graph_converter.batch([c] * count)
        assert (g.n_bonds <= 4096) == (count == 26)
        many = model(g, "efs")
        for i in range(count):
            assert torch.equal(one["e"][0], many["e"][i])
            report(f"merged envelopes {count}/{i}: F", one["f"][0], many["f"][i], 2e-6)
