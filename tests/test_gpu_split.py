"""Contractions whose tiles are cut along K: few tiles and a long contraction,
an unfilled last wave, a last unit shorter than the others. The exact forms
add integers, so that a split result equals the unsplit one bit for bit (whose
accuracy the parity tests hold); the BF16x3 form is compared with the oracle and repeats itself exactly."""
import ctypes

import numpy as np
import pytest
import torch

import muscle_gb300 as m
from muscle_gb300 import _lib
from oracle import muscle_ref as ref
from tests.gpu_util import to_np

pytestmark = pytest.mark.gpu

# (M, N, K, batch): tiles of 128 rows by 32 (BF16x3: 64) embedded columns
SHAPES = [(1, 1, 1000, 1), (5, 7, 4097, 1), (128, 32, 321, 1), (130, 70, 2500, 1), (128, 32, 640, 3),
          (700, 660, 257, 1), (128 * 9, 32 * 17, 96, 1), (33, 20, 70000, 1), (200, 300, 1100, 5)]


def _run(plan, A, B, C, full):
    """The plan with the workspace it asks for, or with the least it accepts
    (found by asking for less), which leaves no room for split tiles."""
    lib = _lib.load()
    need = int(plan.workspace_bytes)
    st = torch.cuda.current_stream().cuda_stream
    ws = torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")
    ws.fill_(255)  # counters and sums start as anything

    def go(nbytes):
        return lib.mgb_contract(plan.handle, A.data_ptr(), B.data_ptr(), C.data_ptr(), ws.data_ptr(), nbytes, st)

    if full:
        assert go(need) == 0
        return need
    lo, hi = 0, need  # the least accepted byte count lies in (lo, hi]
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if go(mid) == 0:
            hi = mid
        else:
            lo = mid
    torch.cuda.synchronize()
    assert go(hi) == 0
    return hi


def _tensors(M, N, K, L, dt):
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K + L)
    A = torch.randn(K, M, L, dtype=dt, device="cuda", generator=g).permute(1, 0, 2)
    B = torch.randn(L, N, K, dtype=dt, device="cuda", generator=g)
    return A, ["i", "k", "l"], B, ["l", "j", "k"], ["i", "j", "l"]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt", [torch.float64, torch.complex128])
@pytest.mark.parametrize("slices", [0, 5, 6, 8])
def test_exact_split_equals_unsplit(shape, dt, slices):
    M, N, K, L = shape
    A, ia, B, ib, ic = _tensors(M, N, K, L, dt)
    out = []
    for full in (True, False):
        C = m.empty_colmajor([M, N, L], dt, "cuda")
        plan = m.contraction_plan(A, ia, B, ib, C, ic, "ozaki", slices)
        used = _run(plan, A, B, C, full)
        torch.cuda.synchronize()
        out.append((to_np(C), used))
    assert m.device_status() == 0
    assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt", [torch.float32, torch.complex64])
def test_bf16x3_split(shape, dt):
    M, N, K, L = shape
    A, ia, B, ib, ic = _tensors(M, N, K, L, dt)
    want = ref.contract(to_np(A).astype(np.complex128 if dt.is_complex else np.float64), ia, to_np(B), ib, ic)
    got = []
    for full in (True, True, False):
        C = m.empty_colmajor([M, N, L], dt, "cuda")
        plan = m.contraction_plan(A, ia, B, ib, C, ic, "bf16x3")
        _run(plan, A, B, C, full)
        torch.cuda.synchronize()
        got.append(to_np(C))
        assert ref.rel_fro(got[-1], want) <= 1e-5
    assert np.array_equal(got[0], got[1])  # whichever unit arrives last
    assert m.device_status() == 0


def test_some_shapes_are_split():
    """The workspace a plan can run with is smaller than the one it asks for
    exactly when tiles are cut."""
    split = []
    for M, N, K, L in SHAPES:
        A, ia, B, ib, ic = _tensors(M, N, K, L, torch.float64)
        C = m.empty_colmajor([M, N, L], torch.float64, "cuda")
        plan = m.contraction_plan(A, ia, B, ib, C, ic, "ozaki", 6)
        split.append(_run(plan, A, B, C, False) < plan.workspace_bytes)
    assert any(split) and not all(split)


def test_split_in_group_and_graph():
    """Split members of a group, alone and replayed from a graph, equal the
    single call bit for bit."""
    items, alone = [], []
    for M, N, K, L in [(5, 7, 4097, 1), (130, 70, 2500, 1), (128, 32, 640, 1), (130, 70, 2500, 1)]:
        for dt in (torch.complex128, torch.complex64):
            A, ia, B, ib, ic = _tensors(M, N, K, L, dt)
            A, B = A[..., 0], B[0]
            C, D = (m.empty_colmajor([M, N], dt, "cuda") for _ in range(2))
            items.append((m.Tensor(C, ["i", "j"]), m.Tensor(A, ["i", "k"]), m.Tensor(B, ["j", "k"])))
            alone.append(m.contract_into(D, ["i", "j"], A, ["i", "k"], B, ["j", "k"]))
    g = m.Group(items)
    for how in ("persistent", "parts", "graph"):
        for c, _, _ in items:
            c.data.fill_(7)
        if how == "graph":
            g.capture().replay()
        else:
            g.execute(parts=1 if how == "persistent" else 2, persistent=how == "persistent")
        torch.cuda.synchronize()
        for (c, a, _), d in zip(items, alone):
            if c.dtype == torch.complex128:
                assert torch.equal(c.data, d)
            else:
                assert torch.linalg.vector_norm(c.data - d) <= 1e-6 * torch.linalg.vector_norm(d)
    assert m.device_status() == 0
