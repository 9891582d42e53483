"""The batch solver that reads the cost blocks once per iteration, at the
edges of its splits: single rows and columns, widths around a vector, a warp
and the widths where more warps share a row, the widest blocks it takes and
one more (the two-pass kernel), batches of one problem (many workers per
problem) and of many tiny ones (many problems per worker), and the cases that
leave its shortcuts.  The reference is the same iteration in float64 torch,
problem by problem.

Tolerances: float64 potentials within 1e-8 of their largest magnitude;
float32 within 2e-5 (exponents reach 72, where one float32 rounding is 4e-6)."""
import math

import numpy as np
import pytest
import torch

from pot_gb300 import _lib, batch as pb

pytestmark = pytest.mark.gpu
F32, F64 = torch.float32, torch.float64


def _batch(rows, cols, dtype, device, seed=0):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    r = lambda *s: torch.rand(*s, generator=g, device=device, dtype=F64)  # noqa: E731
    lay = pb.RaggedLayout(rows, cols, dtype, device)
    Ms, As, Bs = [], [], []
    for n, m in zip(rows, cols):
        x, y = r(int(n), 2), r(int(m), 2)
        Ms.append((0.5 * ((x[:, None] - y[None]) ** 2).sum(2)).to(dtype))
        a, b = r(int(n)) + 0.2, r(int(m)) + 0.2
        As.append((a / a.sum()).to(dtype))
        Bs.append((b / b.sum()).to(dtype))
    return lay, pb.pack_dense(lay, Ms), Ms, As, Bs


def _reference(M, a, b, reg, iters, u, omega=1.0):
    M, la, lb = M.double(), torch.log(a.double()), torch.log(b.double())
    v = None
    for _ in range(iters):
        vn = lb - torch.logsumexp(u[:, None] - M / reg, 0)
        v = vn if v is None or omega == 1.0 else v + omega * (vn - v)
        un = la - torch.logsumexp(v[None, :] - M / reg, 1)
        u = un if omega == 1.0 else u + omega * (un - u)
    return u, v


def _close(x, y, dtype):
    assert torch.equal(torch.isfinite(x), torch.isfinite(y))
    fin = torch.isfinite(y)
    scale = float(y[fin].abs().max().clamp_min(1.0))
    assert float((x.double() - y)[fin].abs().max()) < (1e-8 if dtype == F64 else 2e-5) * scale


BATCHES = {"single": ([1], [1]), "row": ([1, 300], [300, 1]), "one": ([2048], [2048]), "wide": ([70], [2049]),
           "widest": ([40, 21], [16384, 37]), "widest64": ([40, 21], [8192, 37]), "beyond": ([12, 9], [16385, 100]),
           "vectors": (list(range(1, 40)), [5 * k % 131 + 1 for k in range(39)]),
           "tiny": ([3] * 3000, [5] * 3000), "uniform": ([130] * 40, [257] * 40), "halves": ([33, 64, 90], [128, 129, 1025]),
           "ragged": ([701, 32, 999, 64, 5, 1000], [64, 1000, 31, 257, 900, 1000])}


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("name", sorted(BATCHES))
def test_log_and_scaling_forms(cuda, name, dtype):
    rows, cols = BATCHES[name]
    lay, Mp, Ms, As, Bs = _batch(rows, cols, dtype, cuda)
    a, b = torch.cat(As), torch.cat(Bs)
    reg, iters = 0.05, 6
    for scaling in (False, True):
        u, v, st, nit, err, _ = pb.run_multi(lay, Mp, a, b, reg, iters, 0.0, scaling=scaling, tail_problems=-1)
        assert (st == _lib.STATUS_MAXITER).all() and (nit == iters - 1).all()
        if scaling:
            u, v = torch.log(u), torch.log(v)
        for p in range(0, lay.B, max(1, lay.B // 40)):
            n, m = int(rows[p]), int(cols[p])
            ur, vr = _reference(Ms[p], As[p], Bs[p], reg, iters, torch.zeros(n, dtype=F64, device=cuda))
            _close(u[int(lay.r_off_np[p]):int(lay.r_off_np[p]) + n], ur, dtype)
            _close(v[int(lay.c_off_np[p]):int(lay.c_off_np[p]) + m], vr, dtype)


@pytest.mark.parametrize("dtype", [F32, F64])
def test_leaving_the_shortcuts_and_relaxed_updates(cuda, dtype):
    """Zero weights, a far warm start, and over-relaxed updates."""
    rows, cols = [64, 300, 90, 1500], [200, 64, 515, 2500]
    lay, Mp, Ms, As, Bs = _batch(rows, cols, dtype, cuda)
    for k in (0, 3):
        As[k][3], Bs[k][5] = 0.0, 0.0
        As[k], Bs[k] = As[k] / As[k].sum(), Bs[k] / Bs[k].sum()
    a, b = torch.cat(As), torch.cat(Bs)
    for spread, omega in ((0.0, 1.0), (200.0, 1.0), (0.0, 1.3)):
        w = [torch.linspace(-spread, spread, n, device=cuda, dtype=F64) for n in rows]
        u, v, _, _, _, _ = pb.run_multi(lay, Mp, a, b, 0.05, 9, 0.0, warm_u=torch.cat(w).to(dtype), omega=omega,
                                        tail_problems=-1)
        for p, (n, m) in enumerate(zip(rows, cols)):
            if omega != 1.0 and p in (0, 3):
                continue  # relaxing towards -inf is not a number in either
            ur, vr = _reference(Ms[p], As[p], Bs[p], 0.05, 9, w[p], omega)
            _close(u[int(lay.r_off_np[p]):int(lay.r_off_np[p]) + n], ur, dtype)
            _close(v[int(lay.c_off_np[p]):int(lay.c_off_np[p]) + m], vr, dtype)


@pytest.mark.parametrize("joint", [False, True])
def test_stops_and_repeats(cuda, joint):
    """Problems leave at their own check (or all at the largest error's), the
    error is that of the returned pair, and every run gives the same bits."""
    rng = np.random.default_rng(3)
    rows, cols = rng.integers(20, 400, 60), rng.integers(20, 400, 60)
    lay, Mp, Ms, As, Bs = _batch(rows, cols, F64, cuda)
    a, b = torch.cat(As), torch.cat(Bs)
    reg = torch.tensor(rng.uniform(0.01, 0.2, 60), device=cuda)
    runs = [pb.run_multi(lay, Mp, a, b, reg, 5000, 1e-9, joint=joint) for _ in range(3)]
    u, v, st, nit, err, _ = runs[0]
    assert (st == 0).all() and (nit % 10 == 0).all() and float(err.max()) < 1e-9
    assert (len(nit.unique()) == 1) == joint
    for p in range(0, 60, 7):
        n, m = int(rows[p]), int(cols[p])
        up = u[int(lay.r_off_np[p]):int(lay.r_off_np[p]) + n]
        vp = v[int(lay.c_off_np[p]):int(lay.c_off_np[p]) + m]
        P = torch.exp(up[:, None] + vp[None, :] - Ms[p] / reg[p])
        e = float(torch.linalg.vector_norm(P.sum(0) - Bs[p]))
        assert math.isclose(e, float(err[p]), rel_tol=1e-3, abs_tol=1e-14)
    for r in runs[1:]:
        for x, y in zip(r[:5], runs[0][:5]):
            assert torch.equal(x, y)
