"""inca_eval_records_noalloc sets a device up on its first call: later calls of any size load no code and take
no device memory. In a process of its own, where nothing has been loaded before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes, sys
import numpy as np, torch
from inca_parallel_gb300 import _lib
lib = _lib.load()
n, npts = 140000, 257
g = torch.Generator(device="cuda").manual_seed(1)
rand = lambda *shape: torch.rand(*shape, dtype=torch.float64, device="cuda", generator=g)
rec = [rand(n), rand(n) + 0.5, rand(n, 3), torch.zeros(n, 3, dtype=torch.int32, device="cuda"), rand(n, 3, 17)]
pts, out = rand(npts, 3), torch.zeros(npts, dtype=torch.float64, device="cuda")
ptr = lambda t: ctypes.c_void_p(t.data_ptr())

def call(n, npts):
    st = lib.inca_eval_records_noalloc(n, *map(ptr, rec), npts, ptr(pts), ptr(out),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert st == 0, st
    return torch.cuda.mem_get_info()[0]

free = call(3, 2)
assert [call(3, 200), call(n, 100), call(n, npts), call(n, npts)] == [free] * 4
"""


def test_later_calls_take_no_memory():
    from inca_parallel_gb300 import build
    build.build()
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": root})
    assert r.returncode == 0, r.stderr[-2000:]
