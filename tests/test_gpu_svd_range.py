"""The thin SVD over the range of magnitudes: columns whose squared norms and
inner products come close to the smallest normal number, or lie that far apart
within one matrix, are rotated like any others."""
import numpy as np
import pytest
import torch

import muscle_gb300 as m
from tests.gpu_util import to_np
from tests.test_gpu_svd_sizes import _buffers, _check, _rand

pytestmark = pytest.mark.gpu


# one cluster, and the cooperative grid; the entries' squares are 2^-1000 (the
# inner products of nearly orthogonal columns are subnormal) and 2^-1024
# (subnormal themselves, each to 2^-50 of the norms)
@pytest.mark.parametrize("shape", [(12, 8), (40, 33), (300, 40)])
@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("e", [-490, -500, -512])
def test_svd_small_magnitudes(shape, cx, e):
    a = _rand(np.random.default_rng(shape[0] + cx), shape, cx)
    scale = 2.0 ** e
    _, U, S, V, run = _buffers(a * scale)
    run()
    torch.cuda.synchronize()
    _check(a, U, S / scale, V)


@pytest.mark.parametrize("shape", [(12, 6), (300, 6)])
@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("step", [60, 100, 150, 190])
def test_svd_graded_columns(shape, cx, step):
    """Column j is 2^(480 - step j) times a random one. The singular values
    then are the diagonal of R in the QR factorisation of the ungraded
    matrix, scaled like its columns, and the left vectors Q's columns, both to
    a relative 2^(-2 step)."""
    b = _rand(np.random.default_rng(step + cx), shape, cx)
    d = 2.0 ** (480.0 - step * np.arange(shape[1]))
    _, U, S, V, run = _buffers(b * d)
    run()
    torch.cuda.synchronize()
    q, r = np.linalg.qr(b)
    U, s = to_np(U), to_np(S)
    assert np.allclose(s / d, np.abs(np.diag(r)), rtol=1e-13, atol=0.0)
    assert np.linalg.norm(U.conj().T @ U - np.eye(shape[1])) <= 1e-13 * shape[1]
    assert np.allclose(np.abs(np.sum(U.conj() * q, axis=0)), 1.0, rtol=0.0, atol=1e-13)
    assert m.device_status() == 0
