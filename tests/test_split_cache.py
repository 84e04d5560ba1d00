"""CPU: the operand splits that ops.as_split keeps for a weight."""
import torch

from matris_b200 import ops


def test_views_of_one_storage_have_splits_of_their_own():
    w = torch.randn(128, 128)
    a, b = ops.as_split(w), ops.as_split(w.t())
    assert torch.equal(a.w, w) and torch.equal(b.w, w.t()) and torch.equal(b.hi16, w.t().to(torch.bfloat16))
    assert ops.as_split(w) is a and ops.as_split(w.t()) is b
    w.mul_(2.0)  # an update in place is seen
    assert torch.equal(ops.as_split(w).w, w)


def test_an_address_handed_out_again_is_not_taken_for_the_old_weight():
    """A view that SplitWeight has to copy: without the entry's own reference its storage would be free for the next weight."""
    for i in range(50):
        w = torch.randn(128, 256)[:, :128]
        assert torch.equal(ops.as_split(w).w, w), i
        del w
