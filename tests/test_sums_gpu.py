"""Sums that return a value to the caller keep what single precision would
drop: each case has one large term and many that a float32 sum of a few terms
loses next to it."""
import ctypes

import pytest
import torch

from pot_gb300 import _lib
from pot_gb300 import batch as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 8), (40, 256), (8, 1), (512, 37)])
def test_marginals_of_the_total_cost(cuda, n, m):
    """Every row (or column, in runs of eight) holds a 1 and entries of 2^-25:
    sum s log(s / a) with a = 1 is what those add up to."""
    P = torch.full((n, m), 2.0 ** -25, device=cuda)
    if m > 1:
        P[:, 0] = 1.0
    else:
        P[0] = 1.0
    a, b = torch.ones(n, device=cuda), torch.ones(m, device=cuda)
    vals = torch.zeros(2, dtype=torch.float64, device=cuda)
    lib = _lib.load()
    scratch = torch.empty(lib.otg_unbalanced_total_doubles(n, m), dtype=torch.float64, device=cuda)
    out = torch.empty(2, device=cuda)
    for rm1, rm2 in ((1.0, float("inf")), (float("inf"), 1.0)):
        _lib.check(lib.otg_unbalanced_total(_lib.OTG_F32, _lib.ptr(P), n, m, m, _lib.ptr(a), _lib.ptr(b), _lib.ptr(vals), 0.0,
                                            rm1, rm2, _lib.ptr(scratch), _lib.ptr(out), _lib.stream_handle(cuda)), "total")
        s = P.double().sum(1 if rm1 == 1.0 else 0)
        ref = float((s * torch.log(s + 1e-16)).sum())
        assert abs(float(out[1]) - ref) <= 1e-6 * abs(ref) + 1e-15, (rm1, float(out[1]), ref)


@pytest.mark.parametrize("n,m", [(8, 4), (64, 16), (100, 7), (512, 512)])
@pytest.mark.parametrize("method", [_lib.OTG_METHOD_LOG, _lib.OTG_METHOD_KNOPP])
def test_values_of_the_plan(cuda, n, m, method):
    """Zero cost: the plan is the outer product of the scalings, a 1 and
    entries of 2^-25 in every row and column of eight by four."""
    lay = pb.RaggedLayout([n], [m], torch.float32, cuda)
    u, v = torch.full((n,), 2.0 ** -25, device=cuda), torch.full((m,), 2.0 ** -25, device=cuda)
    u[::8], v[::4] = 1.0, 1.0
    a, b = torch.ones(n, device=cuda), torch.ones(m, device=cuda)
    M = torch.full((lay.total_m,), float("inf"), device=cuda)
    lay.block(M, 0).zero_()
    uu, vv = (torch.log(u), torch.log(v)) if method == _lib.OTG_METHOD_LOG else (u, v)
    reg = torch.ones(1, dtype=torch.float64, device=cuda)
    P, vals = pb.batched_plan(lay, M, uu, vv, a, b, reg, method)
    mass = float(lay.block(P, 0).double().sum())
    # next to the rounding of 2^-25 as an exponential, what a float32 sum of 32 entries drops is 1e-6 of the mass
    assert abs(float(vals[0, 2]) - mass) <= 1e-8 * mass
    lg = lay.block(P, 0).double()
    ref = float((lg * torch.log(lg + 1e-16)).sum())
    assert abs(float(vals[0, 1]) - ref) <= 1e-6 * abs(ref)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("m", [1, 5, 7, 8, 1030])
def test_plan_writes_its_columns_only(cuda, dtype, m):
    """Rows of a wider array: what lies behind column m is the caller's."""
    n, ld = 21, (m + 12) // 4 * 4
    one = lambda k, t: torch.tensor([k], dtype=t, device=cuda)  # noqa: E731
    M = torch.rand(n, ld, dtype=dtype, device=cuda)
    P = torch.full((n, ld), -3.0, dtype=dtype, device=cuda)
    u, v, a, b = (torch.zeros(k, dtype=dtype, device=cuda) for k in (n, m, n, m))
    vals, reg, off = torch.empty(3, dtype=torch.float64, device=cuda), one(0.5, torch.float64), one(0, torch.int64)
    rows, cols, ldm = one(n, torch.int32), one(m, torch.int32), one(ld, torch.int32)
    t = _lib.OtgPlanTable(dtype=_lib.dtype_code(dtype), method=_lib.OTG_METHOD_LOG, nprob=1, kl=0, M=M.data_ptr(),
                          m_off=off.data_ptr(), rows=rows.data_ptr(), cols=cols.data_ptr(), ldm=ldm.data_ptr(),
                          r_off=off.data_ptr(), c_off=off.data_ptr(), u=u.data_ptr(), v=v.data_ptr(), a=a.data_ptr(),
                          b=b.data_ptr(), reg=reg.data_ptr(), P=P.data_ptr(), out_vals=vals.data_ptr())
    _lib.check(_lib.load().otg_batched_plan(ctypes.byref(t), n, _lib.stream_handle(cuda)), "plan")
    ref = torch.exp(-M[:, :m].double() / 0.5)
    assert float(((P[:, :m].double() - ref) / ref).abs().max()) < 1e-5
    assert bool((P[:, m:] == -3.0).all())
