"""GPU: the K <= 16 linear layers at row counts around a warp's rows and a resident grid, and at every padding of K."""
import pytest
import torch

from gpu_util import dev, report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rows", [1, 3, 5, 31, 33, 40001])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 16])
def test_small_linear(n_rows, k):
    from matris_b200 import ops
    g = torch.Generator().manual_seed(17 * n_rows + k)
    x, w, dy = (torch.randn(*s, generator=g) for s in ((n_rows, k), (128, k), (n_rows, 128)))
    report(f"forward k={k}", ops.small_linear_fwd(dev(x), dev(w)), x.double() @ w.double().T, 1e-5)
    want = dy.double() @ w.double()
    report(f"backward k={k}", ops.small_linear_bwd(dev(dy), dev(w)), want, 1e-5, scaled=True)
    dx = dev(x.clone())
    ops.small_linear_bwd(dev(dy), dev(w), dx, accumulate=True)
    report(f"backward, accumulated k={k}", dx, x.double() + want, 1e-5, scaled=True)
