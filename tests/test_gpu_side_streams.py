"""GPU: an evaluation whose independent branches run on side streams against the same one on a single stream (which it takes
while every launch is timed), repeated back to back from two caller streams so that buffers are reused at once."""
import pytest
import torch

from gpu_util import report
from matris_b200 import workloads
from matris_b200.weights import random_checkpoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own_buffers", [False, True])
@pytest.mark.parametrize("n_crystals,config", [(1, {}), (24, {}), (3, dict(use_smoothed_for_delta_edge=True)),
                                               (3, dict(graph_conv_mlp="MLP"))])
def test_side_streams_match_one_stream(n_crystals, config, own_buffers, monkeypatch):
    """own_buffers: every buffer from torch's allocator and all internals recomputed, as for a system too large for a workspace"""
    from matris_b200 import MatRIS, _lib
    from matris_b200 import model as model_module
    ck = random_checkpoint(dict(num_layers=2, reference_energy="mpa", **config), seed=5, jitter=0.1)
    model = MatRIS.from_dict(ck).to("cuda")
    if own_buffers:
        monkeypatch.setattr(model_module, "WORKSPACE_LIMIT", 0)
        model.keep_activations = False
    g = model.graph_converter.batch(workloads.random_crystals(n_crystals, seed=2))
    results = lambda o: [o["e"], torch.cat(list(o["f"])), torch.stack(list(o["s"])), torch.cat(list(o["m"]))]
    _lib.profile = []
    try:
        want = [t.clone() for t in results(model(g, task="efsm"))]
    finally:
        _lib.profile = None
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = []
    for i in range(12):
        with torch.cuda.stream(streams[i % 2]):
            got.append([t.clone() for t in results(model(g, task="efsm"))])
    torch.cuda.synchronize()
    for out in got:
        for name, a, b in zip("efsm", out, want):
            report(f"side streams {name}", a, b, 1e-5, scaled=True)
