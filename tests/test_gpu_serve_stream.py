"""A request waits for what its caller's stream has queued before it, the
default stream's work included."""
import pytest
import torch

import muscle_gb300 as m
from muscle_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("default", [True, False])
@pytest.mark.parametrize("form", ["auto", "plain"])
def test_requests_wait_for_the_callers_stream(default, form):
    a, b = (m.Tensor(torch.zeros(64, 64, dtype=torch.float64, device="cuda"), i) for i in (["i", "k"], ["k", "j"]))
    with m.Server(form=form) as server:
        server.submit(a, b).wait()
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.default_stream() if default else torch.cuda.Stream()):
            torch.cuda._sleep(int(4e8))
            a.data.fill_(1.0)
            b.data.fill_(2.0)
            r = server.submit(a, b)
            assert r.wait() == _lib.OK
        torch.cuda.synchronize()
        assert torch.equal(r.out.data, torch.full_like(r.out.data, 128.0))
