"""CPU: what bench.py makes of an instrumented step's records."""
import os
import re

import bench
from conftest import ROOT
from matris_b200._lib import _Elapsed


def contraction_calls():
    """The names under which the evaluation's driver records operations that carry a count of floating-point operations."""
    text = open(os.path.join(ROOT, "matris_b200", "csrc", "evaluate.cu")).read()
    names = set()
    for m in re.finditer(r"R\.op\(", text):
        end, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        name, counts = text[m.end():end - 1].rsplit("}", 1)  # (name, the launch as a lambda, counts ...)
        if counts.count(","):
            names |= set(re.findall(r'"(mb_\w+)"', name))
    return names


def test_every_contraction_counts():
    calls = contraction_calls()
    assert {"mb_gemm", "mb_gated_mlp_fwd", "mb_mlp_bwd_data", "mb_attn_mlp_bwd", "mb_smooth_mlp_bwd", "mb_node_mlp_bwd"} == calls
    records = [(n, _Elapsed(), _Elapsed(2.0), dict(flops=3e9, bytes=5e6, rows=100, k=256, n=256, fused=True)) for n in sorted(calls)]
    records.append(("mb_seg_sum", _Elapsed(), _Elapsed(1.0), None))
    per, shapes, gemm = bench.profile_sums(records)
    assert gemm == dict(flops=18e9, ms=12.0, bytes=30e6, launches=6, calls=sorted(calls))
    assert per["mb_seg_sum"] == [1, 1.0] and per["mb_attn_mlp_bwd"] == [1, 2.0]
    assert shapes == {"gated rows=100 K=256 N=256": [6, 12.0, 18e9]}
