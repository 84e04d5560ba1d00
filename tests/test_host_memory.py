"""CPU: a C entry point that cannot get host memory returns a status (it used to end the process with a C++ exception)."""
import subprocess
import sys

from conftest import ROOT
from matris_b200 import build

CHILD = r"""
import ctypes as C, resource, sys
sys.path.insert(0, sys.argv[1])
from matris_b200 import _lib
lib = _lib.load()
M, layers = _lib.MbModelParams(), (_lib.MbLayerParams * 1)()
M.layers, M.n_layers = layers, 1 << 28  # bookkeeping of gigabytes, asked for before any layer is looked at
e = _lib.MbEval()
e.model = C.pointer(M)
e.n_atoms, e.n_struct, e.n_edges, e.n_bonds, e.n_triplets, e.e = 8, 1, 64, 32, 64, 256
size = C.c_size_t(0)
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (64 << 20), resource.RLIM_INFINITY))
print(lib.mb_evaluate_workspace(C.byref(e), C.byref(size)))
"""


def test_evaluation_without_host_memory_is_a_status():
    build.build()
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "7", (r.returncode, r.stdout, r.stderr[-500:])
