"""contract_into runs in the workspace it is given whenever the plan can run with
that many bytes, and in one of its own otherwise."""
import pytest
import torch

import muscle_gb300 as m
from tests.test_gpu_split import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float64, torch.complex128])
def test_the_least_workspace_is_used(dt):
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(5000, 100, dtype=dt, device="cuda", generator=g).T
    B = torch.randn(20, 5000, dtype=dt, device="cuda", generator=g).T
    C = m.empty_colmajor([100, 20], dt, "cuda")
    args = (C, ["i", "j"], A, ["i", "k"], B, ["k", "j"])
    plan = m.contraction_plan(A, ["i", "k"], B, ["k", "j"], C, ["i", "j"])
    least, full = _run(plan, A, B, C, False), plan.workspace_bytes
    assert least < full
    want = m.contract_into(*args).clone()
    for n, used in ((full, True), (least, True), (least - 1, False), (0, False)):
        ws = torch.full((max(n, 1),), 255, dtype=torch.uint8, device="cuda")[:n]
        C.fill_(7)
        m.contract_into(*args, workspace=ws)
        torch.cuda.synchronize()
        assert torch.equal(C, want)
        if used:
            assert plan.report(ws)["slices"] in range(3, 9)
        else:
            assert bool((ws == 255).all())
