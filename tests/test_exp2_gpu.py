"""The fp64 exponential of the kernels, through the plan kernel with zero
potentials and reg such that the exponent is -M itself: within 0.52 ulp of
the exact value (rounding 0.5, table and series 0.02) plus the reference's
rounding; one unit of the smallest denormal below the normal range."""
import ctypes

import numpy as np
import pytest
import torch

from pot_gb300 import _lib

pytestmark = pytest.mark.gpu


def _exp2(x, device):
    M = torch.tensor(-x, dtype=torch.float64, device=device).reshape(1, -1)
    m = M.shape[1]
    u, v = torch.zeros(1, dtype=torch.float64, device=device), torch.zeros(m, dtype=torch.float64, device=device)
    P = torch.empty_like(M)
    _lib.check(_lib.load().otg_dense_plan(_lib.dtype_code(M.dtype), _lib.OTG_METHOD_LOG, ctypes.c_void_p(M.data_ptr()), 1, m, m,
                                          _lib.ptr(u), _lib.ptr(v), 1.4426950408889634, _lib.ptr(P), m, None,
                                          _lib.stream_handle(device)), "otg_dense_plan")
    return P.cpu().numpy().reshape(-1)


@pytest.mark.parametrize("lo,hi", [(-1.0, 1.0), (-40.0, 40.0), (-1021.9, 1023.9), (-1e-9, 1e-9)])
def test_normal_range(cuda, lo, hi):
    rng = np.random.default_rng(7)
    x = np.concatenate([rng.uniform(lo, hi, 200000), np.linspace(lo, hi, 4097), np.array([lo, hi, 0.0, -0.0])])
    x = np.concatenate([x, np.clip(np.round(x * 256) / 256, lo, hi)])  # the ends of the reduced range
    ref = np.exp2(x.astype(np.longdouble))
    err = np.abs(_exp2(x, cuda).astype(np.longdouble) - ref) / np.spacing(ref.astype(np.float64)).astype(np.longdouble)
    assert float(err.max()) <= 0.55


def test_edges(cuda):
    x = np.array([np.nan, np.inf, -np.inf, 1024.0, 1e300, -1e300, -1100.0, -1075.5, 1023.999, -1022.0, -1021.99999])
    got = _exp2(x, cuda)
    assert np.isnan(got[0]) and got[1] == np.inf and got[2] == 0.0 and got[3] == np.inf and got[4] == np.inf
    assert got[5] == 0.0 and got[6] == 0.0 and got[7] == 0.0
    np.testing.assert_allclose(got[8:], np.exp2(x[8:]), rtol=2.5e-16)
    d = np.linspace(-1074.9, -1022.0, 1000)
    ref = np.exp2(d.astype(np.longdouble))
    # below the normal range the result is rounded twice
    assert float(np.max(np.abs(_exp2(d, cuda).astype(np.longdouble) - ref))) <= 1.01 * 5e-324 + 2.0 ** -1074 * 0.01
