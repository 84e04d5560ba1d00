"""CPU: the native host side of a batch against the same arithmetic in NumPy, bit for bit."""
import numpy as np
import pytest
import torch

from matris_b200 import build, workloads
from matris_b200.graph import HostBatch, cell_grid


@pytest.fixture(scope="module", autouse=True)
def library():
    build.build()


@pytest.mark.parametrize("count,cutoff", [(1, 6.0), (17, 6.0), (40, 1.5)])
def test_host_batch(count, cutoff):
    crystals = workloads.random_crystals(count, seed=11)
    if cutoff < 2:  # long thin cells: the cap on the number of cells is reached
        crystals = [c._replace(lattice=c.lattice @ np.diag([1.0, 9.0, 2.0])) for c in crystals]
    hb = HostBatch([c.numbers for c in crystals], [c.cart for c in crystals], [c.lattice for c in crystals], cutoff, pin=False)
    n = np.array([len(c.numbers) for c in crystals])
    N, B = n.sum(), len(n)
    cart, lat = np.concatenate([c.cart for c in crystals]), np.stack([c.lattice for c in crystals])
    inv, struct = np.linalg.inv(lat), np.repeat(np.arange(B), n)
    frac = np.einsum("ni,nij->nj", cart, inv[struct]).astype(np.float32)
    lat32 = lat.astype(np.float32)
    parts = [struct, np.concatenate([[0], np.cumsum(n)]), hb.i32.numpy()[N + B + 1:N + 9 * B + 1],
             np.concatenate([c.numbers for c in crystals]), np.einsum("ni,nij->nj", frac, lat32[struct]).ravel().view(np.int32),
             lat32.ravel().view(np.int32)]
    want = np.concatenate([np.asarray(p, dtype=np.int32) for p in parts])
    assert np.array_equal(hb.i32.numpy()[:len(want)], want)
    vol = hb.i32.numpy()[len(want):].view(np.float32)
    assert len(vol) == B and np.allclose(vol, np.linalg.det(lat), rtol=1e-5)
    assert np.array_equal(hb.frac32, frac)
    assert torch.equal(hb.f64, torch.from_numpy(np.concatenate([cart.ravel(), lat.ravel(), inv.ravel()])))
    grid, n_cells, volume = cell_grid(lat, n, cutoff)
    cells, half, base = grid[:, 0:3].astype(np.int64), grid[:, 3:6], grid[:, 6]
    width = np.stack([np.abs(np.linalg.det(lat)) / np.linalg.norm(np.cross(lat[:, (k + 1) % 3], lat[:, (k + 2) % 3]), axis=1)
                      for k in range(3)], axis=1)
    assert (cells >= 1).all() and (cells.prod(1) <= np.maximum(4 * n + 8, 1)).all()
    assert np.array_equal(base, np.cumsum(cells.prod(1)) - cells.prod(1)) and n_cells == cells.prod(1).sum()
    assert (half * width / cells >= cutoff * (1 - 1e-9)).all() and ((half - 1) * width / cells < cutoff).all()
    assert np.allclose(volume, np.abs(np.linalg.det(lat)))


def test_singular_lattice():
    with pytest.raises((ValueError, np.linalg.LinAlgError)):
        cell_grid(np.zeros((1, 3, 3)), np.array([2]), 6.0)


@pytest.mark.parametrize("numbers,ok", [([1, 94], True), ([29, 0], False), ([-3, 29], False), ([95, 8], False), ([2 ** 32 + 8, 8], False)])
def test_elements_outside_the_tables_are_refused(numbers, ok):
    """Graphs take any atomic number; a model refuses the ones its tables have no row for (the kernels do not look)."""
    from matris_b200 import MatRIS
    from matris_b200.graph import HostBatch, upload
    model = MatRIS(num_layers=1)
    hb = HostBatch([np.array([6]), np.array(numbers)], [np.zeros((1, 3)), np.eye(2, 3)], [5 * np.eye(3)] * 2, 6.0, pin=False)
    g = upload(hb, 6.0, 4.0, "cpu")
    if ok:
        model._check_elements(g)
    else:
        with pytest.raises(IndexError, match="the model knows the elements 1 to 94"):
            model._check_elements(g)
