"""The dense solver that reads the cost once per iteration, at the edges of
its splits: single rows and columns, widths around a vector and a warp,
batches with a remainder, the border between costs kept in shared memory and
streamed ones, rows that are not whole 16-byte vectors, the widest rows it
takes and one more (the two-pass kernel), and the cases that leave its
shortcuts (zero weights, forbidden entries, far warm starts, small
regularisation).  The reference is the same iteration in float64 torch.

Tolerances: float64 plans within 1e-9 (relative L1) and potentials within
1e-8, the dense parity tests' bounds; float32 plans within 1e-5, potentials
within 1e-5 of their largest magnitude (exponents reach 72 here, where one
float32 rounding is 4e-6)."""
import math

import numpy as np
import pytest
import torch

from pot_gb300 import _lib, bregman

pytestmark = pytest.mark.gpu

LOG, KNOPP, UNB = _lib.OTG_METHOD_LOG, _lib.OTG_METHOD_KNOPP, _lib.OTG_METHOD_UNB
F32, F64 = torch.float32, torch.float64


def _problem(n, m, dtype, device, seed=0):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    r = lambda *s: torch.rand(*s, generator=g, device=device, dtype=F64)  # noqa: E731
    x, y = r(n, 2), r(m, 2)
    M = (x[:, None, 0] - y[None, :, 0]) ** 2 + (x[:, None, 1] - y[None, :, 1]) ** 2
    M = (M / M.max().clamp_min(1e-3)).to(dtype)
    a, b = r(n) + 0.2, r(m) + 0.2
    return M, (a / a.sum()).to(dtype), (b / b.sum()).to(dtype)


def _log_reference(M, a, b, reg, iters, u):
    M, a, b = M.double(), a.double(), b.double()
    for _ in range(iters):
        v = torch.log(b) - torch.logsumexp(u[:, None] - M / reg, 0)
        u = torch.log(a) - torch.logsumexp(v[None, :] - M / reg, 1)
    return u, v


def _unb_reference(M, a, b, reg, reg_m, iters):
    M, a, b = M.double(), a.double(), b.double()
    K = torch.exp(-M / reg) * a[:, None] * b[None, :]
    fi = reg_m / (reg_m + reg)
    v = torch.ones_like(b)
    for _ in range(iters):
        u = (a / (K @ v)) ** fi
        v = (b / (K.T @ u)) ** fi
    return u, v


def _plan(M, u, v, reg):
    return torch.exp(u.double()[:, None] + v.double()[None, :] - M.double() / reg)


def _check(M, u, v, uref, vref, reg, dtype):
    P, Q = _plan(M, u, v, reg), _plan(M, uref, vref, reg)
    assert float((P - Q).abs().sum() / Q.sum()) < (1e-9 if dtype == F64 else 1e-5)
    for x, y in ((u, uref), (v, vref)):
        fin = torch.isfinite(y)
        assert torch.equal(fin, torch.isfinite(x))
        scale = float(y[fin].abs().max().clamp_min(1.0))
        assert float((x.double() - y)[fin].abs().max()) < (1e-8 if dtype == F64 else 1e-5) * scale


SHAPES = [(1, 1), (1, 300), (300, 1), (5, 7), (9, 128), (33, 129), (17, 1023), (150, 1025), (1300, 61), (2600, 96),
          (700, 2049), (2000, 3000), (2200, 4096), (2300, 4099), (40, 8192), (30, 8193), (20, 16384), (12, 16385),
          (9000, 1001)]


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,m", SHAPES)
def test_log_and_scaling_forms(cuda, n, m, dtype):
    M, a, b = _problem(n, m, dtype, cuda)
    reg, iters = 0.05, 7
    u0 = torch.zeros(n, dtype=F64, device=cuda)
    uref, vref = _log_reference(M, a, b, reg, iters, u0)
    r = bregman.solve_dense(M, a, b, reg, LOG, iters, 0.0)
    assert r.status == _lib.STATUS_MAXITER and r.niter == iters - 1 and len(r.errs) == 1
    _check(M, r.u, r.v, uref, vref, reg, dtype)
    for gibbs in ((None, True) if dtype == F64 else (None,)):
        r = bregman.solve_dense(M, a, b, reg, KNOPP, iters, 0.0, gibbs=gibbs)
        _check(M, torch.log(r.u), torch.log(r.v), uref - math.log(n), vref + math.log(n), reg, dtype)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,m", [(1, 5), (33, 129), (700, 2049), (2300, 4099), (9000, 1001), (12, 16385)])
def test_unbalanced_form(cuda, n, m, dtype):
    M, a, b = _problem(n, m, dtype, cuda)
    r = bregman.solve_dense(M, a, b, 0.05, UNB, 9, 0.0, check_period=1, unbalanced=(0.7, 0.7, 0))
    u, v = _unb_reference(M, a, b, 0.05, 0.7, 9)
    tol = 1e-9 if dtype == F64 else 1e-5
    assert float(((r.u.double() - u) / u).abs().max()) < tol
    assert float(((r.v.double() - v) / v).abs().max()) < tol


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,m", [(130, 200), (2300, 4099)])
def test_rows_of_a_wider_buffer(cuda, n, m, dtype):
    """A view with a row stride that is no multiple of 16 bytes."""
    M, a, b = _problem(n, m, dtype, cuda)
    W = torch.full((n, m + 3), -7.0, dtype=dtype, device=cuda)
    W[:, :m] = M
    r0 = bregman.solve_dense(M, a, b, 0.05, LOG, 12, 0.0)
    r1 = bregman.solve_dense(W[:, :m], a, b, 0.05, LOG, 12, 0.0)
    uref, vref = _log_reference(M, a, b, 0.05, 12, torch.zeros(n, dtype=F64, device=cuda))
    _check(M, r0.u, r0.v, uref, vref, 0.05, dtype)
    _check(M, r1.u, r1.v, uref, vref, 0.05, dtype)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,m", [(60, 200), (2300, 4096)])
def test_leaving_the_shortcuts(cuda, n, m, dtype):
    """Zero weights, forbidden entries, a far warm start (row sums and column
    sums far from the previous plan's) and small regularisation."""
    M, a, b = _problem(n, m, dtype, cuda)
    a[3], b[5] = 0.0, 0.0
    a, b = a / a.sum(), b / b.sum()
    M[7, : m // 2] = float("inf")
    for reg, spread in ((0.02, 0.0), (0.02, 200.0), (0.003, 0.0)):
        w = torch.linspace(-spread, spread, n, device=cuda, dtype=F64)
        uref, vref = _log_reference(M, a, b, reg, 14, w)
        r = bregman.solve_dense(M, a, b, reg, LOG, 14, 0.0, w.to(dtype), torch.zeros(m, dtype=dtype, device=cuda))
        P, Q = _plan(M, r.u, r.v, reg), _plan(M, uref, vref, reg)
        # float32: the exponents reach 480, where one rounding is 3e-5
        assert float((P - Q).abs().sum() / Q.sum()) < (1e-9 if dtype == F64 else 1e-3 if reg < 0.01 else 2e-5)
        assert float(r.u[3]) == -math.inf and float(r.v[5]) == -math.inf


def test_error_history_repeats(cuda):
    M, a, b = _problem(2300, 4099, F32, cuda)
    runs = [bregman.solve_dense(M, a, b, 0.02, LOG, 45, 0.0) for _ in range(4)]
    for r in runs[1:]:
        np.testing.assert_array_equal(r.errs, runs[0].errs)
        assert torch.equal(r.u, runs[0].u) and torch.equal(r.v, runs[0].v)
