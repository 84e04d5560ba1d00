"""CPU: what the compiler says of the sources (nvcc cross-compiles without a GPU)."""
import os
import re
import shutil
import subprocess

import pytest

from matris_b200 import build

pytestmark = pytest.mark.skipif(shutil.which(os.environ.get("NVCC", "nvcc")) is None, reason="no CUDA compiler")


def nvcc(source, *flags):
    r = subprocess.run([os.environ.get("NVCC", "nvcc"), *flags, os.path.join(build.CSRC, source), "-o", os.devnull], stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout
    return r.stdout


def test_row_kernels_spill_no_more_than_they_were_measured_with():
    """Kernels whose register limit was chosen with a few spills (the limit's gain is measured beside each): more of them lose it."""
    out = nvcc("rowwise.cu", *build.NVCC_FLAGS, "-c", "-Xptxas=-v")
    spills = {m[0]: int(m[1]) for m in re.findall(r"Compiling entry function '(\S+)'.*?(\d+) bytes spill stores", out, re.S)}
    assert [n for name, n in spills.items() if "21k_smooth_env_bwd_lineE" in name] == [8]


@pytest.mark.parametrize("source", build.SOURCES)
def test_no_warnings(source):
    """The front end has nothing to remark (device code at -O0: the remarks do not depend on it)."""
    out = nvcc(source, "--cuda", "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "-Xcicc", "-O0", "-I", build.INCLUDE, "-I",
               build.CSRC)
    assert "warning" not in out, out
