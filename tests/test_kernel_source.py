"""CPU: rules of the tensor-core kernels that no run can be relied on to show, read from their source."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "matris_b200", "csrc")


def code(name):
    """The source without comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def body(text, start):
    """The braces that open at or after ``start``, with what they hold."""
    i = text.index("{", start)
    depth = 0
    for k in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[i:k + 1]
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("name,n_requests", [("mlp_fused.cuh", 2), ("linear_tma.cuh", 1)])
def test_proxy_fence_before_copies_into_patches_that_threads_stored_to(name, n_requests):
    """A patch that threads fill with ordinary stores (gathered rows, addend sums) and the copy engine fills next: the thread
    that asks for the copy executes a proxy fence first.  An mbarrier orders the threads but not the two proxies."""
    text = code(name)
    requests = [body(text, m.start()) for m in re.finditer(r"auto request = ", text)]
    assert len(requests) == n_requests
    for r in requests:
        assert 0 <= r.find("to_async_proxy()") < r.find("load_patch("), r
