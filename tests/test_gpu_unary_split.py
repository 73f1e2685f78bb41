"""Partial sums with few outputs: every way the terms are shared by threads,
warps and blocks, with and without the workspace for parts, against exact
sums of integers (any order gives the same result) and of Float64 data
against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

import muscle_gb300 as m
from muscle_gb300 import _lib
from oracle import muscle_ref as ref
from tests.gpu_util import to_dev, to_np

pytestmark = pytest.mark.gpu

# shape (labels a, b, c, ...), kept labels
CASES = [((254607,), ""), ((1,), ""), ((31, 33), ""), ((64, 20000), "a"), ((64, 20000), "b"), ((3, 700, 90), "b"),
         ((3, 5, 4099), "b"), ((100000, 3), "b"), ((7, 50000), "a"), ((40, 16, 25), "a"), ((40, 15), "a"),
         ((2, 3, 5, 7, 11, 13), "ace"), ((1025, 2431), "b"), ((1023, 9), "b"), ((129, 8193), "a"), ((33, 1 << 16), "a")]


def _run(X, ix, Y, iy, with_ws):
    lib = _lib.load()
    p = m.unary_plan(X, [m.Index(i) for i in ix], Y, [m.Index(i) for i in iy])
    n = p.workspace_bytes if with_ws else 0
    ws = torch.empty(max(n, 1), dtype=torch.uint8, device="cuda")
    _lib.check(lib.mgb_unary(p.handle, X.data_ptr(), Y.data_ptr(), ws.data_ptr() if n else None, n,
                             torch.cuda.current_stream().cuda_stream), lib)
    torch.cuda.synchronize()
    return n


@pytest.mark.parametrize("shape,keep", CASES)
@pytest.mark.parametrize("dt", [np.float64, np.complex128, np.float32, np.complex64])
def test_integers_are_summed_exactly(shape, keep, dt):
    rng = np.random.default_rng(len(shape) + shape[0])
    x = rng.integers(-3, 4, size=shape).astype(dt)
    if np.issubdtype(dt, np.complexfloating):
        x = (x + 1j * rng.integers(-3, 4, size=shape)).astype(dt)
    ix = [chr(97 + i) for i in range(len(shape))]
    want = x.sum(axis=tuple(i for i, c in enumerate(ix) if c not in keep))
    for order in ("F", "C"):  # the reduced labels fastest, or slowest
        X = to_dev(np.array(x, order=order))
        for with_ws in (True, False):
            Y = m.empty_colmajor([shape[ix.index(c)] for c in keep], X.dtype, "cuda")
            _run(X, ix, Y, list(keep), with_ws)
            assert np.array_equal(to_np(Y), want), (order, with_ws)


@pytest.mark.parametrize("shape,keep", CASES)
@pytest.mark.parametrize("dt", [np.float64, np.complex128])
def test_float_sums(shape, keep, dt):
    rng = np.random.default_rng(3)
    x = rng.standard_normal(shape)
    if dt == np.complex128:
        x = x + 1j * rng.standard_normal(shape)
    ix = [chr(97 + i) for i in range(len(shape))]
    got = m.unary_einsum(m.Tensor(to_dev(np.array(x, order="F")), ix), out=list(keep))
    axes = tuple(i for i, c in enumerate(ix) if c not in keep)
    want = x.sum(axis=axes)
    # one rounding here; numpy's pairwise sum errs by a few ulp of the absolute sum
    assert np.all(np.abs(to_np(got.data) - want) <= 1e-14 * np.abs(x).sum(axis=axes))


def test_infinities_meet_across_parts():
    x = np.ones(300000)
    x[5], x[299990] = np.inf, np.inf
    X = to_dev(x)
    Y = torch.empty((), dtype=torch.float64, device="cuda")
    assert _run(X, ["a"], Y, [], True) > 0
    assert to_np(Y) == np.inf
    X[299990] = -np.inf
    _run(X, ["a"], Y, [], True)
    assert np.isnan(to_np(Y))
