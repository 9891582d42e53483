"""Batched plan kernel at the edges of its vectors, chunks and row groups,
packed as the layout packs and at an odd address.  float32: exponents up to
20 in magnitude carry 2^-24 twice and the exponential 2^-22, together below
4e-6 of an entry, and as much again for the sums' float parts; float64 has
2^-53 in the same places."""
import numpy as np
import pytest
import torch

from pot_gb300 import _lib
from pot_gb300 import batch as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(1, 1)], [(5, 7), (33, 1), (2, 130)], [(33, 1025)], [(9, 4100), (40, 3)]])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kl", [False, True])
@pytest.mark.parametrize("odd", [0, 1])
def test_plan_edges(cuda, sizes, dtype, kl, odd):
    rng = np.random.default_rng(len(sizes) + sizes[0][0])
    lay = pb.RaggedLayout([s[0] for s in sizes], [s[1] for s in sizes], dtype, cuda)
    new = lambda k, lo, hi: torch.tensor(rng.uniform(lo, hi, k), dtype=dtype, device=cuda)  # noqa: E731
    M = new(lay.total_m + odd, 0.0, 1.0)[odd:]
    a, b = new(lay.total_r, 0.1, 1.0), new(lay.total_c, 0.1, 1.0)
    u, v = new(lay.total_r, -1.0, 0.0), new(lay.total_c, -1.0, 0.0)
    reg = torch.full((lay.B,), 0.1, dtype=torch.float64, device=cuda)
    tol = 1e-5 if dtype == torch.float32 else 2e-14
    for method in (_lib.OTG_METHOD_LOG, _lib.OTG_METHOD_KNOPP):
        uu, vv = (u, v) if method == _lib.OTG_METHOD_LOG else (torch.exp(u), torch.exp(v))
        P, vals = pb.batched_plan(lay, M, uu, vv, a, b, reg, method, kl=kl)
        for p, (n, m) in enumerate(sizes):
            C, got = lay.block(M, p).double(), lay.block(P, p).double()
            r0, c0 = int(lay.r_off_np[p]), int(lay.c_off_np[p])
            ud, vd = uu[r0:r0 + n].double(), vv[c0:c0 + m].double()
            if method == _lib.OTG_METHOD_LOG:
                ref = torch.exp(ud[:, None] + vd[None, :] - C / 0.1)
            else:
                ref = ud[:, None] * torch.exp(-C / 0.1) * vd[None, :]
            assert float(((got - ref).abs() / ref).max()) <= tol
            w = a[r0:r0 + n].double()[:, None] * b[c0:c0 + m].double()[None, :] if kl else 1.0
            lg = torch.log(ref / w + 1e-16)
            for x, terms in zip(vals[p].tolist(), (C * ref, ref * lg, ref)):
                assert abs(x - float(terms.sum())) <= tol * float((terms.abs() + ref).sum())
