"""The fp64 power of the unbalanced update, through one iteration over a zero
cost with one column: u_i = a_i^(reg_m / (reg_m + reg)).  Within 0.52 ulp of
the exact value plus the reference's rounding in the normal range; outside it
the library's (two units)."""
import numpy as np
import pytest
import torch

from pot_gb300 import _lib, bregman

pytestmark = pytest.mark.gpu


def _pow(x, rm, reg, device):
    n = len(x)
    M = torch.zeros(n, 1, dtype=torch.float64, device=device)
    a = torch.tensor(x, dtype=torch.float64, device=device)
    b = torch.ones(1, dtype=torch.float64, device=device)
    r = bregman.solve_dense(M, a, b, reg, _lib.OTG_METHOD_UNB, 1, 0.0, check_period=1, unbalanced=(rm, rm, 1))
    return r.u.cpu().numpy()


@pytest.mark.parametrize("rm,reg", [(1.0, 0.05), (0.1, 1.0), (1e6, 0.01), (1e-5, 2.0), (3.0, 3.0)])
def test_power(cuda, rm, reg):
    rng = np.random.default_rng(3)
    x = np.concatenate([np.exp(rng.uniform(-690, 690, 4000)), np.exp(rng.uniform(-3, 3, 4000)), 1 + rng.uniform(-1e-6, 1e-6, 1000),
                        rng.integers(88, 184, 2000) / 128.0, [1.0, np.sqrt(0.5), np.sqrt(2.0), 2.0, 0.5, 2.3e-308, 1.7e308]])
    ref = np.power(x.astype(np.longdouble), np.longdouble(rm / (rm + reg)))
    err = np.abs(_pow(x, rm, reg, cuda).astype(np.longdouble) - ref) / np.spacing(ref.astype(np.float64)).astype(np.longdouble)
    assert float(err.max()) <= 0.55


def test_power_edges(cuda):
    x = np.array([0.0, 5e-324, 1e-310, 2.2250738585072014e-308, 1.0])
    got = _pow(x, 1.0, 1.0, cuda)
    assert got[0] == 0.0 and got[4] == 1.0
    np.testing.assert_allclose(got[1:4], np.sqrt(x[1:4]), rtol=5e-16)
