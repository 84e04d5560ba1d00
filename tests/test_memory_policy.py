"""CPU: how many layers keep their internals - the estimate from two counts against the library's dry run of the same evaluation."""
import ctypes as C

import pytest

from matris_b200 import MatRIS, _lib

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
