"""GPU: sums of row gradients per node / bond / centre atom against index_add in float64."""
import pytest
import torch

from gpu_util import dev, report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_nodes,mean,by_ctr", [(1, 3, False), (7, 40, False), (300, 40, False), (513, 5, False), (513, 5, True)])
def test_seg_sum(n_nodes, mean, by_ctr):
    from matris_b200 import ops
    g = torch.Generator().manual_seed(n_nodes)
    count = torch.randint(0, 2 * mean + 1, (n_nodes,), generator=g)
    count[0] = max(1, int(count[0]))
    tgt = torch.repeat_interleave(torch.arange(n_nodes), count)
    R = len(tgt)
    src = torch.randint(0, n_nodes, (R,), generator=g)
    perm = torch.argsort(src, stable=True)
    tp = torch.cat([torch.zeros(1, dtype=torch.long), count.cumsum(0)])
    sp = torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(src, minlength=n_nodes).cumsum(0)])
    x = torch.randn(R, 256, generator=g)
    n_ctr = 11
    ctr = (tgt * 2 + (torch.arange(R) - tp[tgt] > count[tgt] // 2)) % n_ctr
    acc = torch.randn(n_ctr, 256, generator=g)
    out_c = dev(acc.clone()) if by_ctr else None
    i32 = lambda t: dev(t, torch.int32)  # noqa: E731
    out = ops.seg_sum(n_nodes, i32(tp), i32(sp), i32(perm), dev(x), i32(ctr) if by_ctr else None, out_c)
    z = torch.zeros(n_nodes, 256, dtype=torch.float64)
    want = torch.cat([z.index_add(0, tgt, x.double()), z.index_add(0, src, x.double())], 1)
    report(f"seg_sum nodes={n_nodes}", out, want, 2e-6, scaled=True)
    if by_ctr:
        report("seg_sum by centre", out_c, acc.double().index_add(0, ctr, x.double()), 2e-6, scaled=True)


def test_pair_sum():
    from matris_b200 import ops
    nb = 77
    perm = torch.randperm(2 * nb, generator=torch.Generator().manual_seed(0))
    rev = torch.empty(2 * nb, dtype=torch.long)
    rev[perm[:nb]], rev[perm[nb:]] = perm[nb:], perm[:nb]
    a, b = torch.randn(2 * nb, 256), torch.randn(2 * nb, 256)
    u2d = perm[:nb]
    i32 = lambda t: dev(t, torch.int32)  # noqa: E731
    for second in (None, b):
        out = ops.pair_sum(nb, i32(u2d), i32(rev), dev(a), None if second is None else dev(second))
        want = a[u2d].double() + a[rev[u2d]].double()
        if second is not None:
            want = torch.cat([want, b[u2d].double() + b[rev[u2d]].double()], 1)
        report("pair_sum", out, want, 1e-6, scaled=True)
