"""CPU: the profiler commands recorded under profiles/ are ones that end by themselves: whole steps are captured for durations only, which
ncu takes in one pass; everything else on one kernel and three launches at the most."""
import glob
import os
import re

import pytest

from conftest import ROOT

FILES = sorted(glob.glob(os.path.join(ROOT, "profiles", "*.md")))


def commands(text):
    return re.findall(r"^ +(ncu --(?:[^\n]*\\\n)*[^\n]*)", text, re.M)


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_captures_are_small(path):
    for c in commands(open(path).read()):
        assert "--clock-control none" in c, c
        metrics = re.search(r"--metrics (\S+)", c)
        if metrics and metrics.group(1) == "gpu__time_duration.sum" and "--section" not in c and "--set" not in c:
            continue
        kernel, count = re.search(r'-k regex:("[^"]*"|\S+)', c), re.search(r" -c (\d+)", c)
        # (one kernel is launched by a micro-benchmark; of an evaluation the pattern names one)
        assert kernel and ("|" not in kernel.group(1) or "bench_gemm" in c), c
        assert count and int(count.group(1)) <= 3, c


def test_commands_are_found():
    assert sum(len(commands(open(p).read())) for p in FILES) >= 5
