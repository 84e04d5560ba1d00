"""GPU: the segment softmax and the smooth segment sum at segment lengths around their batches of rows, against float64."""
import pytest
import torch

from gpu_util import dev, report

pytestmark = pytest.mark.gpu


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed))


def _csr(seg, n):
    ptr = torch.zeros(n + 1, dtype=torch.int64)
    ptr[1:] = torch.cumsum(torch.bincount(seg, minlength=n), 0)
    return torch.argsort(seg, stable=True), ptr


@pytest.mark.parametrize("lengths", [[1], [0, 1, 3, 4, 5, 7, 8, 9], [31, 0, 32, 33, 63, 64, 65, 0], [200, 257]])
@pytest.mark.parametrize("with_emap", [False, True])
def test_segment_lengths(lengths, with_emap):
    from matris_b200 import ops
    n, rows = len(lengths), sum(lengths)
    i32 = torch.int32
    g = torch.Generator().manual_seed(rows)
    tgt = torch.repeat_interleave(torch.arange(n), torch.tensor(lengths))
    src = tgt[torch.randperm(rows, generator=g)]
    emap = torch.randint(0, rows, (rows,), generator=g) if with_emap else None
    (_, tptr), (perm, sptr) = _csr(tgt, n), _csr(src, n)
    logits, h, env = 4 * rnd(rows, 256, seed=1), rnd(rows, 128, seed=2), rnd(max(rows, n), 128, seed=3)
    d_emap = dev(emap, i32) if with_emap else None
    agg = ops.seg_attn_fwd(n, dev(tptr, i32), dev(sptr, i32), dev(perm, i32), d_emap, dev(logits), dev(h))[:2]
    L = (logits[emap] if with_emap else logits).double()
    for side, (seg, cols, out) in enumerate(((tgt, L[:, 128:], agg[0]), (src, L[:, :128], agg[1]))):
        ref = torch.zeros(n, 128, dtype=torch.float64)
        for k in range(n):
            if (seg == k).any():
                ref[k] = (torch.softmax(cols[seg == k], 0) * h[seg == k].double()).sum(0)
        report(f"segment softmax side {side}", out, ref, 5e-6)
    smooth = ops.seg_smooth_sum_fwd(n, dev(tptr, i32), d_emap, None if with_emap else dev(src, i32), dev(env), dev(h))
    E = env.double()
    s = E[emap] if with_emap else E[src] * E[tgt]
    report("smooth segment sum", smooth, torch.zeros(n, 128, dtype=torch.float64).index_add_(0, tgt, h.double() * s), 1e-6,
           scaled=True)
    if not with_emap:
        e = E.clone().requires_grad_(True)
        dagg = rnd(n, 128, seed=4)
        out = torch.zeros(n, 128, dtype=torch.float64).index_add(0, tgt, h.double() * e[src] * e[tgt])
        (de,) = torch.autograd.grad((out * dagg.double()).sum(), [e])
        denv = ops.seg_smooth_sum_bwd_env(n, dev(tptr, i32), dev(sptr, i32), dev(perm, i32), dev(tgt, i32), dev(src, i32), None, None,
                                          dev(env), dev(h), dev(dagg))
        report("smooth segment sum: gradient of the envelope", denv, de[:n], 1e-6, scaled=True)


@pytest.mark.parametrize("value", [float("-inf"), -3.4028234663852886e38])
@pytest.mark.parametrize("with_emap", [False, True])
@pytest.mark.parametrize("lengths", [[3, 9], [40, 70, 5]])
def test_rows_masked_with_the_lowest_logits(lengths, with_emap, value):
    """Rows whose logit is -inf or the lowest float drop out of the softmax, also where they fill a whole batch of rows of a warp
    (the first four or eight of a segment, or a later one)."""
    from matris_b200 import ops
    n, rows, i32 = len(lengths), sum(lengths), torch.int32
    tgt = torch.repeat_interleave(torch.arange(n), torch.tensor(lengths))
    (perm, tptr) = _csr(tgt, n)
    emap = torch.arange(rows) if with_emap else None
    logits, h = 4 * rnd(rows, 256, seed=1), rnd(rows, 128, seed=2)
    start = torch.repeat_interleave(tptr[:-1], torch.tensor(lengths))
    at = torch.arange(rows) - start  # position in the segment; its last row always stays
    masked = ((at < 16) | ((at >= 24) & (at < 48))) & (at < torch.tensor(lengths)[tgt] - 1)
    logits[masked, ::2] = value
    agg = ops.seg_attn_fwd(n, dev(tptr, i32), dev(tptr, i32), dev(perm, i32), dev(emap, i32) if with_emap else None, dev(logits),
                           dev(h))[:2]
    for cols, out in ((logits[:, 128:], agg[0]), (logits[:, :128], agg[1])):
        ref = torch.stack([(torch.softmax(cols[tgt == k].double(), 0) * h[tgt == k].double()).sum(0) for k in range(n)])
        report(f"segment softmax, rows masked with {value}", out, ref, 5e-6)
