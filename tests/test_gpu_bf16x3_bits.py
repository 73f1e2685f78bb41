"""Float32 / ComplexF32 results of the BF16x3 form have the same bits however
the contraction is run: alone with the workspace that the plan asks for or
with the least it takes, as an entry of a batch, as a member of a group of any
size, served, and within the fixed scratch of mgb_contract_noalloc."""
import numpy as np
import pytest
import torch

import muscle_gb300 as m
from muscle_gb300 import _lib
from oracle import muscle_ref as ref
from tests.gpu_util import to_np
from tests.test_gpu_split import _run

pytestmark = pytest.mark.gpu

# one tile of many parts; a last part of one chunk, and of a few k; several
# tiles; nearly a wave; a wave and more (one sum); too short for parts
SHAPES = [(100, 20, 20000), (128, 64, 8 * 32 * 17), (60, 50, 8 * 32 * 16 + 5), (300, 200, 3000), (128 * 15, 64 * 10, 2100),
          (128 * 17, 64 * 9, 2100), (128, 64, 100)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt", [torch.float32, torch.complex64])
def test_bits_do_not_depend_on_the_call(shape, dt):
    M, N, K = shape
    L = 40 if M * N < 100000 else 3
    g = torch.Generator(device="cuda").manual_seed(M + K)
    A = torch.randn(L, K, M, dtype=dt, device="cuda", generator=g).permute(2, 1, 0)
    B = torch.randn(L, N, K, dtype=dt, device="cuda", generator=g).permute(2, 1, 0)
    new = lambda: m.empty_colmajor([M, N], dt, "cuda")
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    C = new()
    plan = m.contraction_plan(A[..., 0], ["i", "k"], B[..., 0], ["k", "j"], C, ["i", "j"], "bf16x3")
    _run(plan, A, B, C, True)
    torch.cuda.synchronize()
    want = ref.contract(to_np(A[..., 0]).astype(np.complex128), ["i", "k"], to_np(B[..., 0]), ["k", "j"], ["i", "j"])
    assert ref.rel_fro(to_np(C), want) <= 1e-5
    got = {}
    got["least workspace"] = new()
    _run(plan, A, B, got["least workspace"], False)
    if _run(plan, A, B, new(), False) <= 32 << 20:
        got["noalloc"] = new()
        _lib.check(lib.mgb_contract_noalloc(plan.handle, A.data_ptr(), B.data_ptr(), got["noalloc"].data_ptr(), st), lib)
    D = m.empty_colmajor([M, N, L], dt, "cuda")
    m.contract_into(D, ["i", "j", "l"], A, ["i", "k", "l"], B, ["k", "j", "l"], "bf16x3")
    got["batch"] = D[..., 0]
    T = lambda x, *i: m.Tensor(x, list(i))
    for n in (1, 2, L):
        items = [(T(new(), "i", "j"), T(A[..., l], "i", "k"), T(B[..., l], "k", "j")) for l in range(n)]
        group = m.Group(items, "bf16x3")
        for persistent in (True, False):
            items[0][0].data.fill_(7)
            group.execute(persistent=persistent)
            torch.cuda.synchronize()
            got["group", n, persistent] = items[0][0].data.clone()
        assert all(torch.equal(c.data, D[..., l]) for l, (c, _, _) in enumerate(items))
    a, b = T(A[..., 0], "i", "k"), T(B[..., 0], "k", "j")
    need = sum(x.numel() for x in (a.data, b.data, C)) * C.element_size()
    for budget in (1 << 32, need + int(plan.workspace_bytes) - 1):  # the second without room for parts
        with m.Server(budget, form="bf16x3") as server:
            r = server.submit(a, b)
            if r.wait() == _lib.OK:
                got["served", budget] = r.out.data
            else:  # one sum: there is no smaller workspace
                assert budget < 1 << 32 and r.wait() == _lib.ERR_OUT_OF_MEMORY
    torch.cuda.synchronize()
    for how, c in got.items():
        assert torch.equal(c, C), how
    assert m.device_status() == 0
