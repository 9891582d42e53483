"""Facts and sums of the Gromov-Wasserstein outer loop against PyTorch in
float64 at the edges of tiles and blocks.  Maxima and flags are exact; sums
over positive terms are bounded by the longest chain of additions (20 float32
roundings for alpha and beta, 9 for the plan sums; float64 with room)."""
import numpy as np
import pytest
import torch

from pot_gb300 import gromov as pgw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (31, 33), (32, 64), (257, 100), (1000, 7)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_facts_and_sums(cuda, n, m, dtype):
    rng = np.random.default_rng(n + 7 * m)
    new = lambda *s: torch.tensor(rng.uniform(0.1, 1.0, s), dtype=dtype, device=cuda)  # noqa: E731
    C1, C2, p, q = new(n, n), new(m, m), new(n), new(m)
    C1 = (C1 + C1.T) / 2
    C1[0, 0] = -3.0
    eps = torch.finfo(dtype).eps
    facts, alpha, beta = pgw._facts(C1, C2, p, q, True)
    got = facts.tolist()
    close = torch.allclose(C2, C2.T, atol=1e-10)
    assert got == [3.0, float(C2.max()), float(p.max()), float(q.max()), 1.0, 1.0 if close else 0.0]
    for v, C, w in ((alpha, C1, p), (beta, C2, q)):
        ref = (C.double() ** 2) @ w.double()
        assert float(((v.double() - ref).abs() / ref).max()) <= 20 * eps
    P, G, F = new(n, m), new(n, m), new(n, m)
    for f in (None, F):
        ref = [P.double().sum(), (G.double() * P.double()).sum(), 0.0 if f is None else (f.double() * P.double()).sum()]
        for x, y in zip(pgw._sums(P, G, f).tolist(), ref):
            assert abs(x - float(y)) <= 9 * eps * float(y)


@pytest.mark.parametrize("i,j,x", [(0, 69, 1.1), (69, 0, 1.1), (33, 2, float("nan")), (5, 5, float("nan")), (40, 41, float("inf"))])
def test_one_entry_breaks_the_symmetry(cuda, i, j, x):
    C = torch.ones(70, 70, device=cuda)
    w = torch.ones(70, device=cuda)
    assert pgw._facts(C, C, w, w, True)[0].tolist()[4:] == [1.0, 1.0]
    D = C.clone()
    D[i, j] = x
    got = pgw._facts(C, D, w, w, True)[0].tolist()
    assert got[4:] == [1.0, 0.0]
    assert np.isnan(got[1]) if np.isnan(x) else got[1] == float(D[i, j])
    D[j, i] = D[i, j]
    sym = float(torch.allclose(D, D.T, atol=1e-10))
    assert pgw._facts(C, D, w, w, True)[0].tolist()[5] == sym
