"""Solves of two sizes from several threads, each on a stream of its own: the
launches of one must not depend on what another thread has just set up.  The
sizes of a pair share a kernel instance and need different amounts of shared
memory."""
import ctypes
import threading

import pytest
import torch

from pot_gb300 import _lib

pytestmark = pytest.mark.gpu
CALLS = 3000


def _dense(lib, cuda, n, m):
    M = torch.rand(n, m, device=cuda)
    a, b, u, v = (torch.full((k,), 1 / k, device=cuda) for k in (n, m, n, m))
    wsb = lib.otg_dense_workspace_bytes(_lib.OTG_F32, n, m, 4, 0)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda)
    p = _lib.OtgDenseProblem(dtype=_lib.OTG_F32, method=_lib.OTG_METHOD_LOG, M=M.data_ptr(), n=n, m=m, ldm=m, a=a.data_ptr(),
                             b=b.data_ptr(), reg=0.1, max_iter=1, hist_cap=4, stop_thr=0.0, out_u=u.data_ptr(),
                             out_v=v.data_ptr(), workspace_bytes=wsb)
    ref = ctypes.byref(p)
    return lambda st: lib.otg_sinkhorn_dense(ref, ctypes.c_void_p(ws.data_ptr()), st), (M, a, b, u, v, ws, p), u


def _grad(lib, cuda, n, m):
    f64 = torch.float64
    M = torch.rand(n, m, device=cuda, dtype=f64)
    a, b = (torch.full((k,), 1 / k, device=cuda, dtype=f64) for k in (n, m))
    P = a[:, None] * b[None, :]
    gM, ga, gb = (torch.empty(s, device=cuda, dtype=f64) for s in ((n, m), n, m))
    wsb = lib.otg_sinkhorn_grad_workspace_bytes(n, m)
    ws, info = torch.empty(wsb, dtype=torch.uint8, device=cuda), torch.empty(4, dtype=torch.int32, device=cuda)
    args = [_lib.ptr(P), m, _lib.ptr(M), m, n, m, _lib.ptr(a), _lib.ptr(b), 0.1, 1e-12, 1, _lib.ptr(gM), m, _lib.ptr(ga),
            _lib.ptr(gb), _lib.ptr(ws), wsb, _lib.ptr(info)]
    return lambda st: lib.otg_sinkhorn_grad(*args, st), (M, a, b, P, gM, ga, gb, ws, info), ga


@pytest.mark.parametrize("make,sizes", [(_dense, ((100, 100), (3000, 1000))), (_grad, ((33, 33), (500, 500)))],
                         ids=["dense", "grad"])
def test_launches_from_several_threads(cuda, make, sizes):
    lib = _lib.load()
    torch.manual_seed(0)
    jobs = [make(lib, cuda, *sizes[k % 2]) for k in range(4)]
    main = _lib.stream_handle(cuda)
    want = []
    for call, _, out in jobs:
        _lib.check(call(main), "alone")
        want.append(out.clone())
    torch.cuda.synchronize()
    codes = [set() for _ in jobs]
    streams = [torch.cuda.Stream(cuda) for _ in jobs]

    def work(k):
        call, st = jobs[k][0], ctypes.c_void_p(streams[k].cuda_stream)
        for _ in range(CALLS):
            codes[k].add(call(st))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == [{0}] * 4, codes
    for (_, _, out), w in zip(jobs, want):
        assert torch.equal(out, w)
