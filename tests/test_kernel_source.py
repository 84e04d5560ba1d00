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


def test_proxy_fence_before_matrix_instructions_read_what_threads_stored():
    """The few-row kernel's operands in shared memory are stored by threads: the fence stands between a warp's stores and the arrival
    that lets the matrix instructions read them."""
    text = code("few_rows.cuh")
    arrivals = [m.start() for m in re.finditer(r"mbar_arrive\((?:x|act)_ready", text)]
    assert len(arrivals) == 3  # row gradients, rows read in place, hidden layer
    for at in arrivals:
        before = text[:at]
        stores = max(before.rfind("st.shared"), before.rfind("few_put4(at"))
        assert before.rfind("to_async_proxy()") > stores, text[at - 200:at]


@pytest.mark.parametrize("name,drains", [
    ("mlp_fused.cuh", ["drain_mma(retired, elected);", "drain_copies(w_ready, ML_W_SLOTS, n);",
                       "if (EPI_RES && !alive) drain_copies(my_full, 2, asked);",
                       "if (!alive) drain_copies(my_conv, 1, conv_asked);", "drain_copies(side_full + 16 * pw, 2, side_asked);"]),
    ("linear_tma.cuh", ["drain_mma(retired, elected);", "drain_copies(w_ready, ML_W_SLOTS, n);",
                        "drain_copies(side_full + 16 * lane, 2, n);", "if (!alive) drain_copies(my_conv, 1, conv_asked);"]),
    ("few_rows.cuh", ["drain_mma(retired, elected);", "drain_copies(w_full, (uint32_t)n_slots, asked);"]),
    ("gemm_persistent.cuh", ["drain_mma(retired, elected);", "drain_copies(w_ready, w_period, wu);"]),
    ("gemm.cu", ["drain_copies(w_full, 2, n_loads);", '"bar.arrive 1, 160;"', '"bar.sync 1, 160;"'])])
def test_nothing_is_in_flight_when_a_block_ends(name, drains):
    """After an expired wait a role may leave copies or matrix instructions behind that nobody has waited for: every role that
    issues them waits for its last ones, counted where they are issued.  A role that has itself used all it asked for
    unless its own wait expired may leave the wait out in that case only."""
    lines = [s.strip() for s in code(name).splitlines()]
    for d in drains:
        assert any(s == d or (d.startswith('"') and d in s) for s in lines), d
    # the counts go up where a copy is issued, and nowhere else
    for counter, issue in (("++conv_asked;", "load_patch("), ("side_asked = side_n + 1;", "load_patch(")):
        at = [i for i, s in enumerate(lines) if s == counter]
        assert all(any(issue in s for s in lines[i:i + 5]) for i in at)


def test_no_launch_assumes_a_number_of_multiprocessors():
    """Grids are sized by what the device says; the number of this card's multiprocessors appears in comments only."""
    for name in sorted(os.listdir(CSRC)):
        assert not re.search(r"\b148\b", code(name)), name


def test_side_streams_that_cannot_be_made_leave_no_error_behind():
    """An evaluation runs without side streams when they cannot be created; the error is taken off the thread's record, where
    the check after the first launch would find it."""
    text = code("evaluate.cu")
    taken = body(text, text.index("static bool side_take("))
    assert "cudaGetLastError();" in body(taken, taken.index("auto failed"))
    for call in re.findall(r"cuda(?:Stream|Event)CreateWithFlags[^;]*;", taken):
        assert call.rstrip("; ").endswith("return failed()"), call
