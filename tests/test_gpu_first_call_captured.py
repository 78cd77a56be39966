"""The first labelling call of a process may be part of a stream capture where no count is asked for.  It runs in a
process of its own, after a call of another kind (which sets the memory pool up)."""
import os
import subprocess
import sys

import pytest

pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes
import numpy as np, torch
import oracle
from poutre2_gb300 import _lib
from poutre2_gb300.image import descriptor
L, driver = _lib.load(), ctypes.CDLL("libcuda.so.1")
f = (np.random.default_rng(5).random((90, 130)) < 0.6).astype(np.uint8) * 9
x = torch.from_numpy(f).cuda()
out = torch.full((90, 130), -1, dtype=torch.int64, device="cuda")
convex, h = torch.empty_like(x), _lib.scalar(4, 1)
dx, do, dc = descriptor(x), descriptor(out), descriptor(convex)
assert L.pg_h_convex(ctypes.byref(dx), ctypes.byref(h), 2, ctypes.byref(dc), None) == 0
stream = torch.cuda.Stream()
handle = ctypes.c_void_p(stream.cuda_stream)
torch.cuda.synchronize()
assert driver.cuStreamBeginCapture_v2(handle, 0) == 0  # a global-mode capture
assert L.pg_label_binary(ctypes.byref(dx), 2, ctypes.byref(do), None, handle) == 0, L.pg_last_error()
graph, ready = ctypes.c_void_p(), ctypes.c_void_p()
assert driver.cuStreamEndCapture(handle, ctypes.byref(graph)) == 0 and graph.value
assert driver.cuGraphInstantiateWithFlags(ctypes.byref(ready), graph, ctypes.c_ulonglong(0)) == 0
assert driver.cuGraphLaunch(ready, handle) == 0
torch.cuda.synchronize()
want, n = oracle.label(f, "SESquare2D")
assert np.array_equal(out.cpu().numpy(), want)
count = ctypes.c_int64(-1)
assert L.pg_label_binary(ctypes.byref(dx), 2, ctypes.byref(do), ctypes.byref(count), None) == 0 and count.value == n
"""


def test_labelling_without_a_count():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
