"""GPU: evaluations from several threads, each on a stream of its own."""
import threading

import pytest
import torch

from gpu_util import report
from matris_b200 import workloads
from matris_b200.weights import random_checkpoint

pytestmark = pytest.mark.gpu


def test_threads_on_their_own_streams_agree_with_one_thread():
    from matris_b200 import MatRIS
    ck = random_checkpoint(dict(num_layers=2, reference_energy="mpa"), seed=5, jitter=0.1)
    model = MatRIS.from_dict(ck).to("cuda")
    lists = [workloads.random_crystals(n, seed=n) for n in (1, 3, 9)]
    results = lambda o: [o["e"], torch.cat(list(o["f"])), torch.stack(list(o["s"])), torch.cat(list(o["m"]))]
    want = [[t.cpu() for t in results(model.predict(c, task="efsm"))] for c in lists]
    got, errors = [[] for _ in lists], []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(8):
                    got[i].append([t.cpu() for t in results(model.predict(lists[i], task="efsm"))])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(lists))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for g, w in zip(got, want):
        assert len(g) == 8
        for out in g:
            for name, a, b in zip("efsm", out, w):
                report(f"threads {name}", a, b, 1e-5, scaled=True)


def test_a_thread_that_ends_gives_its_memory_back():
    """The tensor maps a thread has made (about 200 KB) go with it: 400 threads one after another leave less than 60 of them would."""
    import resource

    from matris_b200 import ops
    x, w = torch.randn(256, 128, device="cuda"), ops.SplitWeight(torch.randn(128, 128, device="cuda"))

    def resident():
        return int(open("/proc/self/statm").read().split()[1]) * resource.getpagesize()

    def one():
        with torch.cuda.stream(stream):
            ops.linear(x, w)

    stream, before = torch.cuda.Stream(), 0
    for i in range(440):
        if i == 40:
            before = resident()
        t = threading.Thread(target=one)
        t.start()
        t.join()
    torch.cuda.synchronize()
    grown = resident() - before
    print(f"grown by {grown / 1e6:.1f} MB")
    assert grown < 60 * 200e3
