"""unary_einsum plans with an output of no elements: created, described and run
like any other, whatever the number of terms that each output would have."""
import os
import subprocess
import sys

import pytest
import torch

import muscle_gb300 as m

PY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muscle.jl_gb300", "python")

# in a process of its own: an arithmetic exception in the library ends it
CODE = """
import ctypes, sys
from muscle_gb300 import _lib
lib = _lib.load()
dt = int(sys.argv[1])
for n in (1, 15, 16, 64, 1024, 4096):
    for strides in ([1, 1], [n, 1]):
        x, kx = _lib.make_desc(dt, [0, 1], [0, n], strides)
        y, ky = _lib.make_desc(dt, [0], [0], [1])
        h, info, ws = ctypes.c_void_p(), _lib.PlanInfo(), ctypes.c_uint64(1)
        _lib.check(lib.mgb_unary_plan(ctypes.byref(h), ctypes.byref(x), ctypes.byref(y)), lib)
        _lib.check(lib.mgb_plan_info_get(h, ctypes.byref(info)), lib)
        _lib.check(lib.mgb_plan_workspace_size(h, ctypes.byref(ws)), lib)
        assert ws.value == 0 and info.workspace_bytes == 0
        _lib.check(lib.mgb_unary(h, None, None, None, 0, None), lib)
"""


@pytest.mark.parametrize("dt", [0, 1, 2, 3])
def test_plan_of_an_empty_output(dt):
    r = subprocess.run([sys.executable, "-c", CODE, str(dt)], capture_output=True, text=True,
                       env={**os.environ, "PYTHONPATH": PY})
    assert r.returncode == 0, (r.returncode, r.stderr)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 16, 1024, 4096])
def test_einsum_with_an_empty_output(n):
    for x in (torch.zeros(0, n, 3, dtype=torch.float64, device="cuda"),
              torch.zeros(n, 0, 3, dtype=torch.float64, device="cuda").permute(1, 0, 2)):
        y = m.unary_einsum(m.Tensor(x, ["a", "b", "c"]), out=["a", "c"])
        assert tuple(y.data.shape) == (0, 3)
    torch.cuda.synchronize()
