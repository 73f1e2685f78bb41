"""BF16x3 sums that overflow at the end of a long contraction are infinite,
whether the tile is cut along K or not."""
import numpy as np
import pytest
import torch

import muscle_gb300 as m
from tests.gpu_util import to_np
from tests.test_gpu_split import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float32, torch.complex64])
@pytest.mark.parametrize("K", [40, 2048, 5000])
def test_overflow_in_the_last_terms(dt, K):
    # terms of 1 and, in the last place, of +-2^200 (bf16 holds every operand)
    M, N = 40, 24
    A, B = torch.ones(M, K, dtype=dt, device="cuda"), torch.ones(K, N, dtype=dt, device="cuda")
    A[::2, -1], A[1::2, -1] = 2.0 ** 100, -(2.0 ** 100)
    B[-1, 1:] = 2.0 ** 100
    want = np.where(np.arange(M)[:, None] % 2 == 0, np.inf, -np.inf) * np.ones(N)
    want[:, 0] = K - 1 + np.where(np.arange(M) % 2 == 0, 2.0 ** 100, -(2.0 ** 100))
    for full in (True, False):
        C = m.empty_colmajor([M, N], dt, "cuda")
        plan = m.contraction_plan(A, ["i", "k"], B, ["k", "j"], C, ["i", "j"], "bf16x3")
        _run(plan, A, B, C, full)
        torch.cuda.synchronize()
        got = to_np(C)
        assert np.array_equal(got.real, want.astype(np.float32)), full
        assert not np.iscomplexobj(got) or np.array_equal(got.imag, np.zeros_like(want))
    assert m.device_status() == 0
