"""The one-launch gradients of the Sinkhorn loss (otg_sinkhorn_grad) against
the same conjugate gradients as CPU torch operations, at the edges of the
split: single rows and columns, odd widths, several vectors per thread, rows
of a wider buffer, the widest problem and one more (torch operations), bins
of zero mass.  Both stop at a relative residual of 1e-12; the system's
condition stays below 1e4 here, so gradients agree to 1e-8 of the largest."""
import pytest
import torch

from pot_gb300 import _lib, bregman
from pot_gb300._autograd import implicit_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (1, 9), (9, 1), (33, 47), (500, 500), (201, 513), (300, 1030), (90, 2049),
                                 (700, 4096), (40, 4097)])
@pytest.mark.parametrize("zeros", [False, True])
def test_against_torch_operations(cuda, n, m, zeros):
    g = torch.Generator(device=cuda)
    g.manual_seed(n * 7 + m)
    r = lambda *s: torch.rand(*s, generator=g, device=cuda, dtype=torch.float64)  # noqa: E731
    buf = r(n, m + 1)
    M = buf[:, :m] if m % 2 else buf[:, :m].contiguous()
    a, b = r(n) + 0.3, r(m) + 0.3
    if zeros:
        if min(n, m) < 3:
            pytest.skip("no bin to spare")
        a[1], b[2] = 0.0, 0.0
    a, b = a / a.sum(), b / b.sum()
    s = bregman.solve_dense(M, a, b, 0.5, _lib.OTG_METHOD_LOG, 2000, 1e-13)
    P = torch.exp(s.u[:, None] + s.v[None, :] - M / 0.5)
    got = implicit_grads(P, M, a, b, 0.5)
    ref = implicit_grads(P.cpu(), M.cpu(), a.cpu(), b.cpu(), 0.5)
    for x, y in zip(got, ref):
        assert x.shape == y.shape
        assert float((x.cpu() - y).abs().max()) <= 1e-8 * max(1e-3, float(y.abs().max()))
