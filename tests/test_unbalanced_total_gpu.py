"""Cost and total cost behind an unbalanced solve against float64 sums in
PyTorch, at the edges of the kernels' blocks.  A marginal is off by at most
nine roundings (float sums of eight entries, fp64 beyond), a KL term by its
derivative times that; the result is rounded once more."""
import numpy as np
import pytest
import torch

from pot_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (7, 129), (130, 65), (1000, 257), (9, 1000)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("rm1,rm2", [(0.7, 1.3), (float("inf"), 0.5), (2.0, float("inf")), (float("inf"), float("inf"))])
def test_total(cuda, n, m, dtype, rm1, rm2):
    rng = np.random.default_rng(n + m)
    P = torch.tensor(rng.uniform(0, 1, (n, m)) / (n * m), dtype=dtype, device=cuda)
    a = torch.tensor(rng.dirichlet(np.ones(n)), dtype=dtype, device=cuda) + 1e-4
    b = torch.tensor(rng.dirichlet(np.ones(m)), dtype=dtype, device=cuda) + 1e-4
    vals = torch.tensor([0.3, -0.2], dtype=torch.float64, device=cuda)
    lib = _lib.load()
    scratch = torch.full((lib.otg_unbalanced_total_doubles(n, m),), float("nan"), dtype=torch.float64, device=cuda)
    out = torch.empty(2, dtype=dtype, device=cuda)
    _lib.check(lib.otg_unbalanced_total(_lib.dtype_code(dtype), _lib.ptr(P), n, m, m, _lib.ptr(a), _lib.ptr(b), _lib.ptr(vals),
                                        0.1, rm1, rm2, _lib.ptr(scratch), _lib.ptr(out), _lib.stream_handle(cuda)), "total")
    eps = torch.finfo(dtype).eps
    ref, room = 0.3 - 0.1 * 0.2, 0.0
    for s, w, rm in ((P.double().sum(1), a.double(), rm1), (P.double().sum(0), b.double(), rm2)):
        if np.isfinite(rm):
            lr = torch.log(s / w + 1e-16)
            ref += rm * float((s * lr).sum())
            room += rm * 9 * eps * float((s * (lr.abs() + 1)).sum())
    got = out.double().tolist()
    assert abs(got[0] - 0.3) <= 0.3 * eps
    assert abs(got[1] - ref) <= room + eps * abs(ref) + 1e-15
