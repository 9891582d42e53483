"""The one-read dense solver away from well-filled histograms: empty bins at
small regularisations, bins of every magnitude down to the smallest denormal,
more CTAs than columns over many iterations.  The reference is the same
iteration in float64 torch.

Tolerances: a log-sum-exp update is non-expansive, so the roundings of the
iterations add up.  Exponents reach 4096 in base 2, where one rounding is
4.6e-13 (float64) or 2.4e-4 (float32); 60 iterations with two updates of two
roundings each stay below 1.2e-10 and 0.06, i.e. 1e-8 and 2e-5 of the largest
potential (2500) with room to spare, and plans (float64) within 1e-9."""
import math

import numpy as np
import pytest
import torch

from pot_gb300 import _lib, bregman

pytestmark = pytest.mark.gpu

LOG = _lib.OTG_METHOD_LOG
F32, F64 = torch.float32, torch.float64


def _line(n, m, dtype, device):
    x = torch.arange(n, dtype=F64, device=device) / (n - 1)
    y = torch.arange(m, dtype=F64, device=device) / (m - 1)
    return ((x[:, None] - y[None, :]) ** 2).to(dtype)


def _log_reference(M, a, b, reg, iters, u):
    M, a, b = M.double(), a.double(), b.double()
    for _ in range(iters):
        v = torch.log(b) - torch.logsumexp(u[:, None] - M / reg, 0)
        u = torch.log(a) - torch.logsumexp(v[None, :] - M / reg, 1)
    return u, v


def _check(M, a, b, reg, iters, warm=None):
    n, m, dtype = M.shape[0], M.shape[1], M.dtype
    u0 = torch.zeros(n, dtype=F64, device=M.device) if warm is None else warm
    w = {} if warm is None else {"warm_u": warm.to(dtype), "warm_v": torch.zeros(m, dtype=dtype, device=M.device)}
    uref, vref = _log_reference(M, a, b, reg, iters, u0)
    r = bregman.solve_dense(M, a, b, reg, LOG, iters, 0.0, **w)
    assert r.status == _lib.STATUS_MAXITER
    for x, y, z in ((r.u, uref, a), (r.v, vref, b)):
        assert torch.equal(x == -math.inf, z == 0) and not torch.isnan(x).any()
        fin = torch.isfinite(y)
        assert torch.equal(fin, torch.isfinite(x))
        scale = float(y[fin].abs().max().clamp_min(1.0))
        assert float((x.double() - y)[fin].abs().max()) < (1e-8 if dtype == F64 else 2e-5) * scale
    if dtype == F64:
        P, Q = (torch.exp(p.double()[:, None] + q.double()[None, :] - M / reg) for p, q in ((r.u, r.v), (uref, vref)))
        assert float((P - Q).abs().sum() / Q.sum()) < 1e-9


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("columns", [False, True])
@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("reg", [1e-3, 5e-4, 4e-4])
def test_empty_bins_at_small_regularisation(cuda, reg, dtype, columns, warm):
    """Columns whose nearest rows are all empty: what is left of them in the
    plan of the first potentials is exp(-gap / reg), nothing at all for the
    smaller regularisations."""
    M = _line(100, 100, dtype, cuda)
    a, b = torch.ones(100, dtype=dtype, device=cuda), torch.full((100,), 0.01, dtype=dtype, device=cuda)
    a[:60] = 0.0
    a /= a.sum()
    if columns:
        a, b = b, a
    _check(M, a, b, reg, 60, torch.linspace(-40.0, 40.0, 100, dtype=F64, device=cuda) if warm else None)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,m", [(1000, 900), (2600, 4100)])
@pytest.mark.parametrize("scale", [1.0, 1e9, 1e-9])
def test_bins_of_every_magnitude(cuda, n, m, dtype, scale):
    """Gaussian histograms: every magnitude from the largest bin down to
    denormals and zeros; total masses other than one."""
    def gauss(k, at, sd):
        return torch.tensor(np.exp(-0.5 * ((np.arange(k) - at * k) / sd) ** 2), dtype=F64)
    a, b = gauss(n, 0.1, n / 200), gauss(m, 0.8, m / 150)
    a, b = ((x / x.sum() * scale).to(dtype).to(cuda) for x in (a, b))
    assert float(a.min()) == 0.0 and 0.0 < float(a[a > 0].min()) < torch.finfo(dtype).tiny
    b *= float(a.double().sum() / b.double().sum())
    _check(_line(n, m, dtype, cuda), a, b, 0.01, 25)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,m", [(16384, 32), (10000, 50), (2600, 96), (40000, 3), (6000, 1)])
@pytest.mark.parametrize("method", ["log", "scaling", "unbalanced"])
def test_more_ctas_than_columns(cuda, n, m, dtype, method):
    """CTAs without a column of their own wait for nobody in the merge: many
    iterations, every run the same bits and the right answer."""
    g = torch.Generator(device=cuda)
    g.manual_seed(n + m)
    r = lambda *s: torch.rand(*s, generator=g, device=cuda, dtype=F64)  # noqa: E731
    M = ((r(n, 1) - r(1, m)) ** 2).to(dtype)
    a, b = r(n) + 0.2, r(m) + 0.2
    a, b = (a / a.sum()).to(dtype), (b / b.sum()).to(dtype)
    iters, kw, code = 3000, {}, {"log": LOG, "scaling": _lib.OTG_METHOD_KNOPP, "unbalanced": _lib.OTG_METHOD_UNB}[method]
    if method == "unbalanced":
        kw = {"unbalanced": (0.7, 0.7, 0), "check_period": 1}
    runs = [bregman.solve_dense(M, a, b, 0.05, code, iters, 0.0, **kw) for _ in range(3)]
    for s in runs:
        assert s.status == _lib.STATUS_MAXITER
        assert torch.equal(s.u, runs[0].u) and torch.equal(s.v, runs[0].v)
    u, v = (runs[0].u.double(), runs[0].v.double())
    # both marginals at the fixed point (unbalanced: u = (a / K v)^fi of the plan's own row sums)
    if method == "unbalanced":
        K = torch.exp(-M.double() / 0.05) * a.double()[:, None] * b.double()[None, :]
        fi = 0.7 / 0.75
        x, y = (a.double() / (K @ v)) ** fi, (b.double() / (K.T @ u)) ** fi
    else:
        if method == "scaling":
            u, v = torch.log(u), torch.log(v)
        P = torch.exp(u[:, None] + v[None, :] - M.double() / 0.05)
        x, y, u, v = P.sum(1), P.sum(0), a.double(), b.double()
    tol = 1e-8 if dtype == F64 else 2e-4
    assert float(((x - u) / u).abs().max()) < tol and float(((y - v) / v).abs().max()) < tol


def test_gradient_with_more_ctas_than_columns(cuda):
    from pot_gb300._autograd import implicit_grads
    n, m = 6000, 20
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    r = lambda *s: torch.rand(*s, generator=g, device=cuda, dtype=F64)  # noqa: E731
    M, a, b = r(n, m), r(n) + 0.3, r(m) + 0.3
    a, b = a / a.sum(), b / b.sum()
    s = bregman.solve_dense(M, a, b, 0.5, LOG, 2000, 1e-13)
    P = torch.exp(s.u[:, None] + s.v[None, :] - M / 0.5)
    ref = implicit_grads(P.cpu(), M.cpu(), a.cpu(), b.cpu(), 0.5)
    for _ in range(200):
        got = implicit_grads(P, M, a, b, 0.5)
    for x, y in zip(got, ref):
        assert float((x.cpu() - y).abs().max()) <= 1e-8 * max(1e-3, float(y.abs().max()))


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,m", [(1024, 1024), (3000, 4100), (2300, 2500)])
def test_half_of_the_bins_empty(cuda, n, m, dtype):
    """Empty rows beside full ones in every batch of rows; a forbidden entry
    in an empty row and a row forbidden but for one entry."""
    a, b = torch.ones(n, dtype=F64, device=cuda), torch.ones(m, dtype=F64, device=cuda)
    a[::2], b[1::3] = 0.0, 0.0
    a[17:40] = 0.0
    a, b = (a / a.sum()).to(dtype), (b / b.sum()).to(dtype)
    M = _line(n, m, dtype, cuda)
    M[4, :100] = math.inf
    M[5, :] = math.inf
    M[5, 9] = 0.5
    _check(M, a, b, 0.02, 20)
