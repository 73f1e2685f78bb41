"""Contractions long and large enough for wide tiles (128 x 64) of the exact
form. Its integer sums do not depend on the tiling, and a row's or a column's
digits on nothing else, so that a few rows of the operand, contracted alone in
narrow tiles, give the same bits."""
import pytest
import torch

import muscle_gb300 as m

pytestmark = pytest.mark.gpu


def _run(A, ia, B, ib, ic, slices):
    ext = dict(zip(ia, A.shape)) | dict(zip(ib, B.shape))
    C = m.empty_colmajor([ext[i] for i in ic], A.dtype, "cuda")
    m.contract_into(C, ic, A, ia, B, ib, "ozaki" if slices else "auto", slices)
    return C


# (M, N, K, batch) in the embedded extents: whole tiles; ragged rows, columns
# and k; a last chunk of one k block; tiles cut along K; batch entries
SHAPES = [(128 * 19, 64 * 16, 4096, 1), (128 * 18 + 37, 64 * 15 + 34, 4100, 1), (128 * 38 - 1, 64 * 8 + 2, 4224 - 96, 1),
          (128 * 36, 128, 16384, 1), (128 * 4 + 6, 64 * 8 + 8, 4096, 8)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt,slices", [(torch.float64, 3), (torch.float64, 6), (torch.complex128, 6), (torch.float64, 0)])
def test_wide_tiles_give_the_bits_of_narrow_ones(shape, dt, slices):
    M, N, K, L = shape
    if dt == torch.complex128:
        N, K = N // 2, K // 2
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(L, K, M, dtype=dt, device="cuda", generator=g).permute(2, 1, 0)
    B = torch.randn(L, N, K, dtype=dt, device="cuda", generator=g).permute(2, 1, 0)
    C = _run(A, ["i", "k", "l"], B, ["k", "j", "l"], ["i", "j", "l"], slices)
    rows = 100
    for first in (0, M - rows):
        part = A[first:first + rows, :, :1]
        one = [_run(part, ["i", "k", "l"], B[:, :, :1], ["k", "j", "l"], ["i", "j", "l"], s)
               for s in ([slices] if slices else [6, 7, 8, 5, 4, 3])]
        assert any(torch.equal(C[first:first + rows, :, :1], c) for c in one)
