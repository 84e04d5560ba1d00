"""CPU: how many layers keep their internals - the estimate from two counts against the library's dry run of the same evaluation."""
import ctypes as C
import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from matris_b200 import MatRIS, _lib, build


@pytest.fixture(scope="module", autouse=True)
def library():
    build.build()


# per atom: directed edges within 6 A, triplets (sparse and dense crystals, close-packed metals)
SHAPES = {"crystals": (28.0, 72.0), "glass": (50.0, 215.0), "bcc": (64.0, 260.0), "perovskite": (69.0, 322.0), "fcc": (78.0, 306.0)}


def dry_run(keep, n_atoms, n_struct, n_edges, n_triplets, n_layers=10):
    """Bytes an evaluation of all outputs needs (the counts alone matter: no device is touched)."""
    M, layers = _lib.MbModelParams(), (_lib.MbLayerParams * n_layers)()
    M.layers, M.n_layers = layers, n_layers
    e = _lib.MbEval()
    e.model = C.pointer(M)
    e.n_atoms, e.n_struct, e.n_edges, e.n_bonds, e.n_triplets = n_atoms, n_struct, n_edges, n_edges // 2, n_triplets
    e.keep_layers, e.f, e.s, e.m = keep, 256, 256, 256
    size = C.c_size_t(0)
    assert _lib.load().mb_evaluate_workspace(C.byref(e), C.byref(size)) == 0
    return size.value


@pytest.mark.parametrize("shape", list(SHAPES))
def test_estimate_is_on_the_safe_side(shape):
    model = MatRIS(num_layers=10)
    for n in (100, 4000, 40000):
        edges, trips = int(SHAPES[shape][0] * n) // 2 * 2, int(SHAPES[shape][1] * n)
        for avail in (5e9, 20e9, 60e9, 180e9):
            k = model.kept_layers(trips, edges, avail)
            assert 0 <= k <= 10
            assert k == 0 or dry_run(k, n, max(1, n // 36), edges, trips) <= 0.9 * avail, (shape, n, avail, k)


def test_keep_activations_overrides_the_estimate():
    model = MatRIS(num_layers=4)
    assert model.kept_layers(1000, 400, 1e12) == 4 and model.kept_layers(10 ** 9, 4 * 10 ** 8, 1e9) == 0
    for keep, want in ((True, 4), (False, 0), (2, 2), (9, 4), (-1, 0)):
        model.keep_activations = keep
        assert model.kept_layers(10 ** 9, 4 * 10 ** 8, 1e9) == want


def batch_of(n_per, edges_per_atom, triplets_per_atom):
    """The parts of a batch's graph that a memory plan reads."""
    ap = np.concatenate([[0], np.cumsum(n_per)])
    ep, tp = 2 * (np.asarray(ap * edges_per_atom, dtype=np.int64) // 2), np.asarray(ap * triplets_per_atom, dtype=np.int64)
    return SimpleNamespace(device=torch.device("cpu"), n_struct=len(n_per), n_atoms=int(ap[-1]), n_edges=int(ep[-1]),
                           n_triplets=int(tp[-1]), structure_slices=lambda: (ap, ep, ep // 2, tp))


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("gigabytes", [4.0, 20.0, 120.0])
def test_sub_batches_and_evaluation_plan_with_the_same_need(shape, gigabytes):
    """A list is cut exactly when the dry run of its batch does not fit with all layers kept, and every part does fit then."""
    model = MatRIS(num_layers=10)
    model._available_bytes = lambda: gigabytes * 1e9
    rng = np.random.default_rng(0)
    per_atom, one = SHAPES[shape], dry_run(10, 4000, 100, int(SHAPES[shape][0] * 4000) // 2 * 2, int(SHAPES[shape][1] * 4000)) / 4000
    for share in (0.8, 0.97, 1.1, 2.5):  # of what fits at once
        n_per = rng.integers(8, 65, max(2, int(share * 0.9 * gigabytes * 1e9 / one / 36.5)))
        g = batch_of(n_per, *per_atom)
        ranges = model.split_for_memory(g)
        fits = dry_run(10, g.n_atoms, g.n_struct, g.n_edges, g.n_triplets) <= 0.9 * gigabytes * 1e9
        assert (ranges == [(0, g.n_struct)]) == fits, (share, ranges)
        ap, ep, _, tp = g.structure_slices()
        assert ranges[0][0] == 0 and ranges[-1][1] == g.n_struct and all(x[1] == y[0] for x, y in zip(ranges, ranges[1:]))
        for a, b in ranges:
            need = dry_run(10, int(ap[b] - ap[a]), b - a, int(ep[b] - ep[a]), int(tp[b] - tp[a]))
            assert need <= 0.9 * gigabytes * 1e9 * (1.0 if fits else 0.93)
        # no more parts than the memory asks for, but for the balancing
        whole = dry_run(10, g.n_atoms, g.n_struct, g.n_edges, g.n_triplets)
        assert fits or len(ranges) <= math.ceil(whole / (0.93 * 0.9 * gigabytes * 1e9)) + 2


@pytest.mark.parametrize("bonds,at_once", [(4096, True), (4097, False), (7123, False), (8192, False)])
def test_envelopes_of_all_layers_are_held_at_once_for_few_bonds_only(bonds, at_once):
    """One launch for all layers' envelopes pays for small graphs; from 4,400 bonds on it costs about 1 % of an evaluation.  Seen in the
    memory of an evaluation that keeps nothing, by the number of layers."""
    few, many = (dry_run(0, 400, 1, 2 * bonds, 2 * bonds, n_layers=n) for n in (10, 20))
    rows = (many - few - 10 * 512 * 2 * 400) / (10 * 512 * bonds)  # a layer's rows of 512 bytes for a bond and its two triplets
    assert 10 <= rows < 10.5 if at_once else 8 <= rows < 8.5  # its features and, at once, two envelopes


def layer_workspace(kind, line, bonds):
    """Bytes a sub-block's forward and backward pass takes: the atom graph of ``bonds`` bonds, or a line graph with two triplets each."""
    rows = 2 * bonds
    g = _lib.MbRowGraph(n_rows=rows, n_nodes=bonds if line else 10, n_edge_rows=rows if line else bonds, n_ctr=10 if line else 0,
                        is_atom=int(not line))
    need, any_ = C.c_size_t(0), 256
    if kind == "attention":
        status = _lib.load().mb_attention_layer(C.byref(_lib.MbAttnParams()), C.byref(g), *[any_] * 2, None, None, *[any_] * 4, None,
                                                C.byref(need), None)
    else:
        atom = any_ if line else None
        status = _lib.load().mb_refine_layer(C.byref(_lib.MbRefineParams()), C.byref(g), *[any_] * 3, atom, None, None, *[any_] * 5, atom,
                                             None, C.byref(need), None)
    assert status == 0
    return need.value


@pytest.mark.parametrize("kind,line,bonds,rows", [("attention", False, 8192, 24), ("attention", False, 16384, 24),
                                                  ("refine", False, 8192, 23), ("refine", False, 16384, 24),
                                                  ("refine", True, 8192, 29), ("refine", True, 16384, 30)])
def test_nothing_is_reserved_that_no_kernel_writes(kind, line, bonds, rows):
    """Rows of 512 bytes a bond.  The sums of a bond's two directed rows have no buffer of their own (they are formed on the way into
    their contraction, or laid where dz2 was), and the envelopes' gradient none where it goes straight on (8,192 bonds)."""
    assert rows <= layer_workspace(kind, line, bonds) / (512 * bonds) < rows + 0.1
