"""The one-read batch solver on histograms of every magnitude (Gaussian tails
down to denormals and zeros, total masses other than one), with empty bins,
and batches that mix them with well-filled problems.  The reference is the
same iteration in float64 torch, problem by problem; the tolerances are those
of test_multi_fused_gpu.py (potentials relative to their largest magnitude)."""
import numpy as np
import pytest
import torch

from pot_gb300 import _lib, batch as pb

pytestmark = pytest.mark.gpu
F32, F64 = torch.float32, torch.float64


def _gauss(k, at, sd, mass):
    x = np.exp(-0.5 * ((np.arange(k) - at * k) / (sd * k)) ** 2)
    return torch.tensor(x / x.sum() * mass)


def _reference(M, a, b, reg, iters):
    M, la, lb = M.double(), torch.log(a.double()), torch.log(b.double())
    u = torch.zeros_like(la)
    for _ in range(iters):
        v = lb - torch.logsumexp(u[:, None] - M / reg, 0)
        u = la - torch.logsumexp(v[None, :] - M / reg, 1)
    return u, v


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("anderson", [0, 3])
def test_tails_and_empty_bins(cuda, dtype, anderson):
    rows, cols = [300, 900, 64, 515, 200, 700], [200, 64, 515, 2500, 200, 600]
    mass = [1.0, 1e9, 1e-9, 1.0, 1.0, 1.0]
    lay = pb.RaggedLayout(rows, cols, dtype, cuda)
    Ms, As, Bs = [], [], []
    for p, (n, m) in enumerate(zip(rows, cols)):
        x, y = (torch.arange(k, dtype=F64, device=cuda) / (k - 1) for k in (n, m))
        Ms.append(((x[:, None] - y[None, :]) ** 2).to(dtype))
        if p < 4:
            a, b = _gauss(n, 0.2, 0.01, mass[p]), _gauss(m, 0.7, 0.012, mass[p])
        else:
            a, b = torch.ones(n, dtype=F64), torch.ones(m, dtype=F64)
            if p == 5:
                a[::2], b[1::3] = 0.0, 0.0
            a, b = a / a.sum(), b / b.sum()
        As.append(a.to(dtype).to(cuda))
        Bs.append(b.to(dtype).to(cuda))
    iters = 12
    u, v, st, nit, err, _ = pb.run_multi(lay, pb.pack_dense(lay, Ms), torch.cat(As), torch.cat(Bs), 0.02, iters, 0.0,
                                         tail_problems=-1, anderson=anderson)
    assert (st == _lib.STATUS_MAXITER).all()
    for p, (n, m) in enumerate(zip(rows, cols)):
        up = u[int(lay.r_off_np[p]):int(lay.r_off_np[p]) + n].double()
        vp = v[int(lay.c_off_np[p]):int(lay.c_off_np[p]) + m].double()
        if anderson:  # (mixing of -inf is not a number: only problems with full histograms; u is the exact row update of v)
            if p != 4:
                continue
            ur, vr = torch.log(As[p].double()) - torch.logsumexp(vp[None, :] - Ms[p].double() / 0.02, 1), vp
        else:
            ur, vr = _reference(Ms[p], As[p], Bs[p], 0.02, iters)
        for x, y in ((up, ur), (vp, vr)):
            assert torch.equal(torch.isfinite(x), torch.isfinite(y))
            fin = torch.isfinite(y)
            assert float((x - y)[fin].abs().max()) < (1e-8 if dtype == F64 else 2e-5) * float(y[fin].abs().max().clamp_min(1.0))
