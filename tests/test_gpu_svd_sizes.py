"""The thin SVD at the edges of its split over the GPU: one column, one pair,
an odd padding column, one cluster with one to four pairs per CTA or a
cooperative grid, columns that fill one to eight registers per thread or are
read again, and more pairs than SMs. Singular values against
LAPACK, reconstruction, orthonormality; extreme magnitudes; graph capture."""
import ctypes

import numpy as np
import pytest
import torch

import muscle_gb300 as m
from tests.gpu_util import to_dev, to_np

pytestmark = pytest.mark.gpu


def _rand(rng, shape, cx):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cx else x


def _buffers(a):
    from muscle_gb300 import _lib

    mm, nn = a.shape
    k, cx = min(mm, nn), np.iscomplexobj(a)
    tdt = torch.complex128 if cx else torch.float64
    U, V = m.empty_colmajor([mm, k], tdt, "cuda"), m.empty_colmajor([nn, k], tdt, "cuda")
    S = torch.empty(k, dtype=torch.float64, device="cuda")
    wsb = ctypes.c_uint64(0)
    lib = _lib.load()
    dt = _lib.C64 if cx else _lib.F64
    _lib.check(lib.mgb_svd_workspace_size(dt, mm, nn, ctypes.byref(wsb)), lib)
    ws = torch.empty(wsb.value, dtype=torch.uint8, device="cuda")
    A = to_dev(np.asfortranarray(a))

    def run():
        _lib.check(lib.mgb_svd(dt, mm, nn, A.data_ptr(), mm, U.data_ptr(), S.data_ptr(), V.data_ptr(), 0, 0,
                               ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), lib)

    return A, U, S, V, run


def _check(a, U, S, V):
    """Backward error and orthogonality of one-sided Jacobi grow with the
    column length through the rotations' rounding: 1e-13 (a few hundred
    ulp) relative, per column for the orthogonality."""
    U, s, V = to_np(U), to_np(S), to_np(V)
    k = min(a.shape)
    want = np.linalg.svd(a, compute_uv=False)
    assert np.all(s[:-1] >= s[1:]) and np.allclose(s, want, rtol=1e-13, atol=1e-13 * want[0])
    assert np.linalg.norm((U * s) @ V.conj().T - a) <= 1e-13 * np.linalg.norm(a)
    assert np.linalg.norm(U.conj().T @ U - np.eye(k)) <= 1e-13 * k
    assert np.linalg.norm(V.conj().T @ V - np.eye(k)) <= 1e-13 * k
    assert m.device_status() == 0


@pytest.mark.parametrize("shape", [(1, 1), (2, 2), (3, 3), (5, 2), (7, 6), (31, 33), (32, 32), (65, 34), (128, 128),
                                   (256, 128), (257, 128), (129, 129), (256, 255), (511, 512), (3000, 7), (310, 310),
                                   (700, 650)])
@pytest.mark.parametrize("cx", [False, True])
def test_svd_split_edges(shape, cx):
    a = _rand(np.random.default_rng(7 * shape[0] + shape[1] + cx), shape, cx)
    _, U, S, V, run = _buffers(a)
    run()
    torch.cuda.synchronize()
    _check(a, U, S, V)


@pytest.mark.parametrize("scale", [2.0 ** -250, 2.0 ** 250])
def test_svd_extreme_magnitudes(scale):
    a = _rand(np.random.default_rng(5), (40, 33), True) * scale
    _, U, S, V, run = _buffers(a)
    run()
    torch.cuda.synchronize()
    _check(a / scale, U, S / scale, V)


def test_svd_under_capture():
    """Captured once, replayed on other values: every replay clears the
    waiting state of the launch."""
    rng = np.random.default_rng(11)
    a = _rand(rng, (48, 64), True)
    A, U, S, V, run = _buffers(a)
    run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        run()
    for _ in range(3):
        a = _rand(rng, (48, 64), True)
        A.copy_(to_dev(np.asfortranarray(a)))
        g.replay()
        torch.cuda.synchronize()
        _check(a, U, S, V)
