"""GPU: neighbour lists around and above the number that an atom's single search keeps on chip (128), bit for bit as the oracle's."""
import numpy as np
import pytest

from matris_b200 import workloads
from test_gpu_graph import check_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a", [3.6, 3.05, 2.2])  # about 78, 128 and 340 neighbours
def test_neighbours_per_atom(a):
    crystals = [workloads.cu_fcc(reps, a=a, sigma=0.12, seed=s) for s, reps in enumerate([(1, 1, 1), (2, 2, 2), (3, 2, 1)])]
    check_batch(crystals + [workloads.demo_pu4si6()], lc=2.6)
