"""Wide tiles (128 x 64) with batch entries, in groups, and with ragged rows and
columns: shapes that the rule sends there, as the plan reports, give the bits
of a few rows contracted alone in narrow tiles."""
import pytest
import torch

import muscle_gb300 as m

pytestmark = pytest.mark.gpu

# (M, N, K, batch) in the embedded extents: batch entries of whole and of cut
# tiles, ragged; ragged rows and columns, few columns in the last tile; the same
# of one wave and more, uncut
SHAPES = [(128 * 3 - 1, 64 * 5 + 34, 9000, 16), (128 * 2 - 5, 64 * 4 - 20, 12000, 24), (128 * 5 - 20, 64 * 9 - 10, 8000, 7),
          (128 * 38 - 91, 64 * 16 + 2, 4128, 1), (128 * 19 - 3, 64 * 24 - 8, 3000, 1)]
IDX = (["i", "k", "l"], ["k", "j", "l"], ["i", "j", "l"])


def _plan(A, B, C, slices):
    ia, ib, ic = (x[:t.dim()] for x, t in zip(IDX, (A, B, C)))
    return m.contraction_plan(A, ia, B, ib, C, ic, "ozaki", slices)


def _run(A, B, slices):
    """The result, the plan's tiling and the slice count that ran."""
    C = m.empty_colmajor([A.shape[0], B.shape[1], *A.shape[2:]], A.dtype, "cuda")
    plan = _plan(A, B, C, slices)
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    ia, ib, ic = (x[:A.dim()] for x in IDX)
    m.contract_into(C, ic, A, ia, B, ib, "ozaki", slices, workspace=ws)
    return C, plan.tiling, slices or plan.report(ws)["slices"]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt,slices", [(torch.float64, 3), (torch.float64, 6), (torch.complex128, 6), (torch.float64, 0)])
def test_wide_tiles_with_batch_entries(shape, dt, slices):
    M, N, K, L = shape
    if dt == torch.complex128:
        N, K = N // 2, K // 2
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(L, K, M, dtype=dt, device="cuda", generator=g).permute(2, 1, 0)
    B = torch.randn(L, N, K, dtype=dt, device="cuda", generator=g).permute(2, 1, 0)
    C, tiling, ran = _run(A, B, slices)
    assert tiling["wide"] and ran in (3, 6)
    for rows in (slice(0, 100), slice(M - 100, M)):
        for l in (0, L - 1):
            want, narrow, S = _run(A[rows, :, l], B[:, :, l], ran)
            assert not narrow["wide"] and S == ran
            assert torch.equal(C[rows, :, l], want)
    if L > 1:  # the same entries as members of a group: a bucket's own launch, and the persistent one
        items = [(m.Tensor(m.empty_colmajor([M, N], dt, "cuda"), ["i", "j"]), m.Tensor(A[..., l], ["i", "k"]),
                  m.Tensor(B[..., l], ["k", "j"])) for l in range(L)]
        group = m.Group(items, "ozaki", slices)
        for persistent in (False, True):
            for parts in (1, 2):
                for c, _, _ in items:
                    c.data.fill_(7)
                group.execute(parts=parts, persistent=persistent)
                torch.cuda.synchronize()
                assert all(torch.equal(c.data, C[..., l]) for l, (c, _, _) in enumerate(items)), (persistent, parts)
    assert m.device_status() == 0


def test_reported_tilings():
    """Short or few tiles run narrow; the plain form has none."""
    new = lambda *s: torch.empty(*s[::-1], dtype=torch.float64, device="cuda").T
    a, b, c = new(100, 2000), new(2000, 16), new(100, 16)
    t = _plan(a, b, c, 6).tiling
    assert not t["wide"] and t["splits"][0] > 1 and t["splits"][1] == 0
    plain = m.contraction_plan(a, ["i", "k"], b, ["k", "j"], c, ["i", "j"], "plain").tiling
    assert plain == {"wide": False, "splits": (0, 0)}
