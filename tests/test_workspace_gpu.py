"""Scratch of the dense solvers: none for what a call does not run, and a
solve that has no room for the one-read kernel's copies takes the two-pass
kernel instead of failing."""
import pytest
import torch

import pot_gb300 as pg
from pot_gb300 import _lib, bregman

pytestmark = pytest.mark.gpu
N, M = 2300, 4099  # streamed rows that are not whole 16-byte vectors


def _problem(cuda, dtype):
    g = torch.Generator(device=cuda)
    g.manual_seed(1)
    C = torch.rand(N, M, generator=g, device=cuda, dtype=dtype)
    a, b = torch.full((N,), 1 / N, device=cuda, dtype=dtype), torch.full((M,), 1 / M, device=cuda, dtype=dtype)
    return C, a, b


def test_stabilised_form_has_no_copy_of_the_cost(cuda):
    C, a, b = _problem(cuda, torch.float32)
    r = bregman.solve_dense(C, a, b, 0.1, _lib.OTG_METHOD_STAB, 20, 0.0, tau=1e3)
    assert r.workspace.numel() < 4 * N * M


def test_float64_scaling_form_has_one_copy_of_the_kernel(cuda):
    C, a, b = _problem(cuda, torch.float64)
    r = bregman.solve_dense(C, a, b, 0.1, _lib.OTG_METHOD_KNOPP, 20, 0.0, read_back=False)
    held = r.workspace.numel() + (0 if r.K is None else r.K.numel() * 8)
    assert held < 1.9 * 8 * N * M


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("method", ["sinkhorn", "sinkhorn_log", "unbalanced"])
def test_without_room_for_the_copy(cuda, monkeypatch, dtype, method):
    C, a, b = _problem(cuda, dtype)

    def solve():
        if method == "unbalanced":
            return pg.sinkhorn_unbalanced(a, b, C, 0.1, 1.0, numItermax=20, stopThr=0.0)
        return pg.sinkhorn(a, b, C, 0.1, method=method, numItermax=20, stopThr=0.0, warn=False)
    want = solve()
    empty = torch.empty
    refused = []

    def no_room(*size, **kw):
        if kw.get("dtype") == torch.uint8 and size and isinstance(size[0], int) and size[0] >= C.numel() * C.element_size():
            refused.append(size[0])
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)
    monkeypatch.setattr(torch, "empty", no_room)
    got = solve()
    assert refused
    tol = 1e-10 if dtype == torch.float64 else 1e-5
    assert float((got.double() - want.double()).abs().sum() / want.double().sum()) < tol


def test_large_workspaces_are_given_back(cuda):
    C, a, b = _problem(cuda, torch.float64)
    before = torch.cuda.memory_allocated(cuda)
    P, log = pg.sinkhorn(a, b, C, 0.1, method="sinkhorn_log", numItermax=20, stopThr=0.0, warn=False, log=True)
    r = bregman.solve_dense(C, a, b, 0.1, _lib.OTG_METHOD_LOG, 20, 0.0)
    assert len(r.errs) == 2 and len(log["err"]) == 2
    held = torch.cuda.memory_allocated(cuda) - before
    assert held < P.numel() * 8 + (8 << 20)
