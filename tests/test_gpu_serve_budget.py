"""What a request is charged: the least workspace its plan runs with while
others wait for the budget, and room for split tiles out of what is free, within a
sixteenth of the budget."""
import time

import pytest
import torch

import muscle_gb300 as m
from muscle_gb300 import _lib
from tests.test_gpu_split import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float64, torch.complex64])
def test_budget_holds_requests_by_their_least_workspace(dt):
    a = m.Tensor(torch.randn(4096, 100, dtype=dt, device="cuda").T, ["i", "k"])
    b = m.Tensor(torch.randn(20, 4096, dtype=dt, device="cuda").T, ["k", "j"])
    c = m.Tensor(m.empty_colmajor([100, 20], dt, "cuda"), ["i", "j"])
    plan = m.contraction_plan(a.data, a.inds, b.data, b.inds, c.data, c.inds)
    resident = sum(t.data.numel() for t in (a, b, c)) * a.data.element_size()
    least, full = _run(plan, a.data, b.data, c.data, False), int(plan.workspace_bytes)
    assert least < full
    want = m.binary_einsum(a, b).data
    n = 24

    def held(server, count):
        """Bytes held by `count` requests that wait for the stream, once all have started
        (or have not after a second)."""
        server.submit(a, b).wait()  # tables and scratch are there
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(int(3e9))
            reqs = [server.submit(a, b, wait_for_stream=True) for _ in range(count)]
        t0 = time.time()
        while server.stats()["pending"] and time.time() - t0 < 1.0:
            time.sleep(0.01)
        s = server.stats()
        for r in reqs:
            assert r.wait() == _lib.OK and torch.equal(r.out.data, want)
        return s["pending"], s["used_bytes"]

    with m.Server((n + 2) * (resident + least), streams=n) as server:
        pending, used = held(server, n)
        assert pending == 0 and used <= (n + 2) * (resident + least)
    with m.Server(1 << 33, streams=n) as server:
        assert held(server, n) == (0, n * (resident + full))
    assert m.device_status() == 0
