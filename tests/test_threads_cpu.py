"""CPU: host state that evaluations in several threads must not share."""
import contextlib
import threading
from types import SimpleNamespace

import torch

from matris_b200 import MatRIS, ops


def test_an_evaluation_leaves_other_threads_their_streams(monkeypatch):
    """While one thread is inside ``forward``, launches of another thread go to that thread's current stream."""
    current = threading.local()
    monkeypatch.setattr(ops, "_raw_stream", lambda device: getattr(current, "stream", 0))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(ops, "gemm_status_async", lambda flag: None)
    monkeypatch.setattr(MatRIS, "device", property(lambda self: torch.device("cuda", 0)))
    model = MatRIS(num_layers=1)
    model._gemm_flag = torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(model, "_as_batch", lambda graphs: SimpleNamespace(device=torch.device("cuda", 0), number_range=(1, 8)))
    inside, leave, seen = threading.Event(), threading.Event(), {}

    def evaluate(g, task):
        seen["evaluating"] = ops._stream()
        inside.set()
        leave.wait(10)
        return {}

    monkeypatch.setattr(model, "_evaluate", evaluate)

    def first():
        current.stream = 111
        model(None)

    t = threading.Thread(target=first)
    t.start()
    assert inside.wait(10)
    current.stream = 222
    seen["other"] = ops._stream()
    leave.set()
    t.join()
    assert seen == {"evaluating": 111, "other": 222}
