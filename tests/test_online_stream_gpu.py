"""Shifted-sum passes of the online Sinkhorn at the edges of their tiles,
row pairs and cluster ranges, against float64 log-sum-exps in PyTorch after a
fixed number of iterations.  The plan's relative L1 distance is bounded by
2e-5, as for every online solve (float32 potentials, dot products of about 22
bits)."""
import numpy as np
import pytest
import torch

from pot_gb300.empirical import online_sinkhorn

pytestmark = pytest.mark.gpu


# one tile and one row block, tiles and row blocks made of padding only
# (n <= 128, m % 256 == 1), rows of one pair shared by every range (few rows,
# many columns), ranges of many row pairs (many rows, few columns), ranges
# that end inside a row pair; both plane widths
@pytest.mark.parametrize("n,m,d", [(1, 1, 3), (128, 257, 16), (129, 256, 17), (256, 512, 64), (100, 20001, 40),
                                   (20001, 100, 12), (3000, 2777, 64), (2561, 4099, 5)])
def test_stream_edges(cuda, n, m, d):
    rng = np.random.default_rng(n + m + d)
    X = torch.tensor(rng.standard_normal((n, d)), dtype=torch.float32, device=cuda)
    Y = torch.tensor(rng.standard_normal((m, d)) * 0.8, dtype=torch.float32, device=cuda)
    a = torch.tensor(rng.dirichlet(np.full(n, 50.0)), dtype=torch.float32, device=cuda)
    b = torch.tensor(rng.dirichlet(np.full(m, 50.0)), dtype=torch.float32, device=cuda)
    C = torch.cdist(X.double(), Y.double(), compute_mode="donot_use_mm_for_euclid_dist") ** 2
    reg, iters = 0.3 * float(C.mean()), 12
    f, g, st, nit, errs = online_sinkhorn(X, Y, reg, a, b, iters, 0.0)
    la, lb = a.double().log(), b.double().log()
    fr, gr = torch.zeros(n, dtype=torch.float64, device=cuda), torch.zeros(m, dtype=torch.float64, device=cuda)
    for _ in range(iters):
        fr = la - torch.logsumexp(gr[None, :] - C / reg, 1)
        gr = lb - torch.logsumexp(fr[:, None] - C / reg, 0)
    P = torch.exp(f.double()[:, None] + g.double()[None, :] - C / reg)
    Pr = torch.exp(fr[:, None] + gr[None, :] - C / reg)
    rel = float((P - Pr).abs().sum() / Pr.sum())
    print("n=%d m=%d d=%d: plan rel L1 %.2e" % (n, m, d, rel))
    assert rel <= 2e-5
