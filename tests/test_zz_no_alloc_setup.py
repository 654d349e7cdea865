"""ndb_b200_run_noalloc sets itself up in the first call on a device, n = 0 included; the
calls after it allocate neither device nor pinned host memory.  In a process of its own:
the set-up happens once per process."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, importlib
import torch
from torch.profiler import ProfilerActivity, profile
pkg = importlib.import_module("nextdbscan-exa_b200")
f = pkg.lib.load().ndb_b200_run_noalloc
f.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32, ctypes.c_float, ctypes.c_int32, ctypes.c_uint32,
              ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
x = torch.rand(5000, 3, device="cuda")
nn, ci = (torch.empty(5000, dtype=torch.int32, device="cuda") for _ in range(2))
torch.cuda.synchronize()
assert f(None, 0, 3, 1.0, 4, 0, None, None, None, None) == 0
with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
    st = f(x.data_ptr(), 5000, 3, 0.1, 4, 0, nn.data_ptr(), ci.data_ptr(), None, None)
    torch.cuda.synchronize()
assert st == 0
names = {e.name for e in p.events()}
assert "cudaLaunchKernel" in names, "the profiler saw no call of the library"
bad = sorted(n for n in names if n.startswith(("cudaMalloc", "cudaHost", "cudaFree")))
assert not bad, bad
"""


def test_only_the_first_call_allocates():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=280)
    assert r.returncode == 0, r.stderr[-2000:]
