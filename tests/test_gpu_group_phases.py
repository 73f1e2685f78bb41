"""A group's two phases by themselves: after one pre-pass the tensor-core phase
may run any number of times, into the outputs as they are now."""
import pytest
import torch

import muscle_gb300 as m
from muscle_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,form,slices", [(torch.float64, "ozaki", 6), (torch.float64, "ozaki", 0),
                                            (torch.complex128, "ozaki", 0), (torch.complex64, "bf16x3", 0)])
def test_finish_may_be_repeated(dt, form, slices):
    # one long tile, two tiles, several waves with an unfilled last one, a short one
    g = torch.Generator(device="cuda").manual_seed(3)
    items = []
    for M, N, K in [(100, 20, 5000), (200, 32, 2500), (128 * 20, 32 * 9, 1200), (64, 16, 40)]:
        A = torch.randn(K, M, dtype=dt, device="cuda", generator=g).T
        B = torch.randn(N, K, dtype=dt, device="cuda", generator=g).T
        items.append((m.Tensor(m.empty_colmajor([M, N], dt, "cuda"), ["i", "j"]), m.Tensor(A, ["i", "k"]),
                      m.Tensor(B, ["k", "j"])))
    group = m.Group(items, form, slices)
    lib = _lib.load()
    st = torch.cuda.current_stream().cuda_stream
    ws, wsb = group.workspace.data_ptr(), group.workspace_bytes
    group.workspace.fill_(255)
    _lib.check(lib.mgb_group_prepare_part(group.handle, 0, 1, ws, wsb, st), lib)
    first = None
    for _ in range(3):
        for c, _, _ in items:
            c.data.fill_(7)
        _lib.check(lib.mgb_group_finish(group.handle, ws, wsb, st), lib)
        torch.cuda.synchronize()
        out = [c.data.clone() for c, _, _ in items]
        if first is None:
            first = out
            for (c, a, b), o in zip(items, out):
                want = a.data.to(torch.complex128) @ b.data.to(torch.complex128)
                err = torch.linalg.vector_norm(o - want) / torch.linalg.vector_norm(want)
                assert err <= (1e-5 if dt == torch.complex64 else 1e-12)
        assert all(torch.equal(x, y) for x, y in zip(out, first))
    assert m.device_status() == 0
