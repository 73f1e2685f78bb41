"""Contraction plans with extents of zero, one and a few: created and described
in every form and element type, alone and with batch labels."""
import os
import subprocess
import sys

import pytest

PY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "muscle.jl_gb300", "python")

# in a process of its own: an arithmetic exception in the library ends it
CODE = """
import ctypes, itertools, sys
from muscle_gb300 import _lib
lib = _lib.load()
dt = int(sys.argv[1])
def desc(modes, ext):
    strides, s = [], 1
    for e in ext:
        strides.append(s)
        s *= max(e, 1)
    return _lib.make_desc(dt, modes, ext, strides)
for M, N, K, L in itertools.product((0, 1, 5, 300), (0, 1, 40), (0, 1, 33, 5000), (None, 0, 1, 3)):
    b = [] if L is None else [L]
    (da, ka), (db, kb), (dc, kc) = (desc([0, 2, 3][:2 + len(b)], [M, K] + b), desc([2, 1, 3][:2 + len(b)], [K, N] + b),
                                    desc([0, 1, 3][:2 + len(b)], [M, N] + b))
    for form, slices in ((0, 0), (1, 0), (2, 0), (2, 3), (2, 6), (3, 0)):
        h, info, ws = ctypes.c_void_p(), _lib.PlanInfo(), ctypes.c_uint64(0)
        st = lib.mgb_contraction_plan(ctypes.byref(h), ctypes.byref(da), ctypes.byref(db), ctypes.byref(dc), form, slices)
        if st:
            assert form in (2, 3), (M, N, K, L, form, st)  # a form that the element type does not have
            continue
        _lib.check(lib.mgb_plan_info_get(h, ctypes.byref(info)), lib)
        _lib.check(lib.mgb_plan_workspace_size(h, ctypes.byref(ws)), lib)
        assert ws.value == info.workspace_bytes and info.m * info.n >= 0
        wide, splits = ctypes.c_int32(0), (ctypes.c_int32 * 2)()
        _lib.check(lib.mgb_plan_tiling(h, ctypes.byref(wide), splits), lib)
        lib.mgb_plan_destroy(h)
"""


@pytest.mark.parametrize("dt", [0, 1, 2, 3])
def test_plans_of_any_extents(dt):
    r = subprocess.run([sys.executable, "-c", CODE, str(dt)], capture_output=True, text=True,
                       env={**os.environ, "PYTHONPATH": PY})
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["float32", "float64", "complex64", "complex128"])
def test_empty_sums_and_outputs(dt):
    import torch

    import muscle_gb300 as m

    t = lambda i, *s: m.Tensor(torch.ones(s, dtype=getattr(torch, dt), device="cuda"), i)
    items = []
    for M, N, K in ((300, 40, 0), (5, 4, 0), (0, 4, 7), (5, 0, 2000), (0, 0, 0)):
        a, b = t(["i", "k"], M, K), t(["k", "j"], K, N)
        c = m.binary_einsum(a, b)
        assert tuple(c.data.shape) == (M, N) and not c.data.any()
        items.append((t(["i", "j"], M, N), a, b))
    m.Group(items).execute()
    torch.cuda.synchronize()
    assert not any(c.data.any() for c, _, _ in items) and m.device_status() == 0
