"""Many long one-tile contractions in one launch, whose cuts along K are
thinned out or dropped by their number: the bits of the single calls, in a group
and in a served batch. Few beside a large one, and the last part of one k."""
import pytest
import torch

import muscle_gb300 as m
from muscle_gb300 import _lib

pytestmark = pytest.mark.gpu


def _items(dt, n, K0):
    g = torch.Generator(device="cuda").manual_seed(n + K0)
    new = lambda *s: torch.randn(*s, dtype=dt, device="cuda", generator=g).T
    shapes = [(90 + i // 32, 12, K0 + 33 * (i % 32)) for i in range(n)] + [(128 * 9, 32 * 17, 96), (128, 16, 32 * 25 + 1)]
    return [(m.Tensor(m.empty_colmajor([M, N], dt, "cuda"), ["i", "j"]), m.Tensor(new(K, M), ["i", "k"]),
             m.Tensor(new(N, K), ["k", "j"])) for M, N, K in shapes]


@pytest.mark.parametrize("n,K0", [(2, 6000), (30, 2000), (170, 1500), (400, 1200)])
@pytest.mark.parametrize("dt,slices", [(torch.float64, 6), (torch.float64, 0), (torch.complex128, 7), (torch.complex64, 0)])
def test_bits_of_single_calls(dt, slices, n, K0):
    items = _items(dt, n, K0)
    want = []
    for c, a, b in items:
        want.append(m.contract_into(torch.empty_like(c.data), ["i", "j"], a.data, ["i", "k"], b.data, ["k", "j"],
                                    "auto", slices))
    group = m.Group(items, "auto", slices)
    for _ in range(2):
        for c, _, _ in items:
            c.data.fill_(7)
        group.execute()
        torch.cuda.synchronize()
        assert all(torch.equal(c.data, w) for (c, _, _), w in zip(items, want))
    with m.Server(slices=slices, max_batch=1024) as server:
        reqs = [server.submit(a, b) for _, a, b in items]
        for r, w in zip(reqs, want):
            assert r.wait() == _lib.OK and torch.equal(r.out.data, w)
    assert m.device_status() == 0
