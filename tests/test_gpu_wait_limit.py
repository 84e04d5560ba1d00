"""GPU: the bound of the kernels' waits is the time the header states."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_wait_gives_up_after_its_limit():
    """A barrier nothing arrives at: the wait lasts the two seconds of its limit and at most a fraction of that longer (the length
    of the hardware's last parked poll and of a launch)."""
    from matris_b200 import ops
    assert ops.gemm_status() == 0
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record()
    ops.selftest_wait_expiry()
    t1.record()
    torch.cuda.synchronize()
    assert ops.gemm_status() == 1 and ops.gemm_status() == 0
    print(f"the wait took {t0.elapsed_time(t1):.1f} ms")
    assert 1999.0 <= t0.elapsed_time(t1) <= 2500.0
