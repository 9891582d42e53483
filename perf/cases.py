"""The calls whose time is measured, and the inputs they are measured on.

Every case is one public entry point as a user's program calls it:

  dense       ``sinkhorn`` on a stored cost: scaling and log-domain form, float32 and float64
  unbalanced  ``sinkhorn_unbalanced`` (KL marginal penalties)
  grad        ``sinkhorn2`` and the gradients of its loss (a training step's forward and backward)
  batch       ``solve_batch``: many equal problems, the whole batch stopping together
  ragged      ``batch.solve_sample_ragged``: point clouds of uneven sizes, each problem stopping on its own
  pairs       ``warmstart.pipeline.solve_cloud_pairs``: equal-size cloud pairs, warm-started
  lazy        ``empirical_sinkhorn(isLazy=True)``: the cost rebuilt from the points in every pass
  egw         ``gromov.entropic_gromov_wasserstein`` in float32

Iterative solves run either to a tolerance that the inputs' precision reaches
with room to spare or for the number of iterations that the caller asks for.
"""
import math

import numpy as np
import torch

import pot_gb300 as pg
from pot_gb300 import batch as pb
from pot_gb300.warmstart import pipeline as wp

_DT = {"f32": torch.float32, "f64": torch.float64}


def listed():
    return [
        # a histogram-sized problem, the library's documentation and test size: latency and launches
        {"name": "dense_f64_100", "kind": "dense", "method": "sinkhorn", "dtype": "f64", "n": 100, "m": 100,
         "reg": 0.05, "iters": 1000, "tol": 1e-9},
        # the usual CPU benchmark of the library: n = m = 1024, float64, default method and threshold
        {"name": "dense_f64_1024", "kind": "dense", "method": "sinkhorn", "dtype": "f64", "n": 1024, "m": 1024,
         "reg": 0.05, "iters": 1000, "tol": 1e-9},
        # small regularisation in double precision needs the log-domain form; sizes that nothing divides
        {"name": "log_f64_777x1001", "kind": "dense", "method": "sinkhorn_log", "dtype": "f64", "n": 777, "m": 1001,
         "reg": 0.02, "iters": 1000, "tol": 1e-9},
        # a single-precision training or matching step with a fixed number of iterations, rows not 16-byte aligned
        {"name": "log_f32_3001x4099", "kind": "dense", "method": "sinkhorn_log", "dtype": "f32", "n": 3001,
         "m": 4099, "reg": 0.02, "iters": 50, "tol": 0.0},
        # a large stored cost (1 GiB): the passes over it are the time
        {"name": "log_f32_16384", "kind": "dense", "method": "sinkhorn_log", "dtype": "f32", "n": 16384, "m": 16384,
         "reg": 0.02, "iters": 30, "tol": 0.0},
        # unequal masses (outlier-robust matching): the unbalanced scaling form
        {"name": "unbalanced_f32_2000x3000", "kind": "unbalanced", "dtype": "f32", "n": 2000, "m": 3000, "reg": 0.05,
         "reg_m": 1.0, "iters": 100, "tol": 0.0},
        # a loss layer: Sinkhorn loss of a mini-batch with gradients of the cost and of both histograms
        {"name": "grad_f64_500", "kind": "grad", "method": "sinkhorn", "dtype": "f64", "n": 500, "m": 500,
         "reg": 0.05, "iters": 1000, "tol": 1e-9},
        # many medium problems in one call, default stop rule of the batched solver
        {"name": "batch_f32_128x512", "kind": "batch", "dtype": "f32", "B": 128, "n": 512, "m": 512, "reg": 0.05,
         "iters": 1000, "tol": 1e-5},
        # a batch of point clouds of uneven sizes (documents, molecules), small to large regularisation
        {"name": "ragged_f32_256", "kind": "ragged", "dtype": "f32", "B": 256, "lo": 32, "hi": 1024, "sizes": 0, "d": 3,
         "reg_lo": 0.01, "reg_hi": 0.1, "iters": 2000, "tol": 1e-6},
        # equal-size cloud pairs at the size of the repository's benchmark, its defaults
        {"name": "pairs_f32_256x2048", "kind": "pairs", "B": 256, "n": 2048, "m": 2048, "d": 16, "reg": 0.02},
        # clouds whose cost matrix is never stored
        {"name": "lazy_f32_16384_d64", "kind": "lazy", "n": 16384, "m": 16384, "d": 64, "reg": 0.1, "iters": 30},
        # matching two metric spaces: tensor products and inner solves in turn
        {"name": "egw_f32_2048", "kind": "egw", "n": 2048, "m": 2048, "eps": 0.02, "outer": 4, "inner": 50},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_float(rng, lo, hi):
    return float("%.3g" % math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["dense", "dense", "dense", "unbalanced", "grad", "batch", "ragged", "pairs", "lazy", "egw"])
    if kind == "dense":
        dtype = rng.choice(["f32", "f64"])
        method = rng.choice(["sinkhorn", "sinkhorn_log"])
        top = 16384 if dtype == "f32" else 2048
        c = {"kind": kind, "method": method, "dtype": dtype, "n": _log_int(rng, 32, top), "m": _log_int(rng, 32, top),
             "reg": _log_float(rng, 0.02, 0.2)}
        if dtype == "f32":
            return dict(c, iters=rng.randint(10, 30), tol=0.0)
        return dict(c, iters=1000, tol=1e-9)
    if kind == "unbalanced":
        dtype = rng.choice(["f32", "f64"])
        top = 8192 if dtype == "f32" else 2048
        return {"kind": kind, "dtype": dtype, "n": _log_int(rng, 32, top), "m": _log_int(rng, 32, top),
                "reg": _log_float(rng, 0.02, 0.2), "reg_m": _log_float(rng, 0.1, 10.0), "iters": rng.randint(20, 100),
                "tol": 0.0}
    if kind == "grad":
        return {"kind": kind, "method": rng.choice(["sinkhorn", "sinkhorn_log"]), "dtype": "f64",
                "n": _log_int(rng, 32, 1024), "m": _log_int(rng, 32, 1024), "reg": _log_float(rng, 0.05, 0.5),
                "iters": 1000, "tol": 1e-9}
    if kind == "batch":
        n, m = _log_int(rng, 16, 1024), _log_int(rng, 16, 1024)
        return {"kind": kind, "dtype": rng.choice(["f32", "f32", "f64"]), "B": max(2, min(512, _log_int(
            rng, 4, max(5, (1 << 26) // (n * m))))), "n": n, "m": m, "reg": _log_float(rng, 0.02, 0.2),
            "iters": 1000, "tol": 1e-5}
    if kind == "ragged":
        return {"kind": kind, "dtype": "f32", "B": _log_int(rng, 16, 256), "lo": 32, "hi": _log_int(rng, 100, 1024),
                "sizes": rng.randint(1, 1 << 20), "d": rng.choice([2, 3, 5, 8, 16]), "reg_lo": 0.01, "reg_hi": 0.1, "iters": 2000, "tol": 1e-6}
    if kind == "pairs":
        return {"kind": kind, "B": _log_int(rng, 8, 256), "n": _log_int(rng, 512, 2048), "m": _log_int(rng, 512, 2048),
                "d": rng.choice([2, 3, 8, 16]), "reg": 0.02}
    if kind == "lazy":
        return {"kind": kind, "n": _log_int(rng, 500, 16384), "m": _log_int(rng, 500, 16384),
                "d": _log_int(rng, 3, 64), "reg": _log_float(rng, 0.05, 0.3), "iters": rng.choice([10, 20, 30])}
    return {"kind": kind, "n": _log_int(rng, 100, 2048), "m": _log_int(rng, 100, 2048),
            "eps": _log_float(rng, 0.02, 0.1), "outer": rng.randint(2, 4), "inner": 50}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _cloud(g, count, n, d, comps=4):
    """count clouds of n points, mixtures of `comps` isotropic Gaussians."""
    mean = torch.randn(count, comps, d, generator=g, device="cuda", dtype=torch.float64)
    std = 0.2 + 0.4 * torch.rand(count, comps, generator=g, device="cuda", dtype=torch.float64)
    k = torch.randint(0, comps, (count, n), generator=g, device="cuda")
    mu = torch.gather(mean, 1, k[..., None].expand(count, n, d))
    return mu + torch.gather(std, 1, k)[..., None] * torch.randn(count, n, d, generator=g, device="cuda",
                                                                 dtype=torch.float64)


def _cost(x, y):
    """Squared distances over their maximum, (B, n, m)."""
    c = (x * x).sum(2)[:, :, None] + (y * y).sum(2)[:, None, :] - 2.0 * x @ y.transpose(1, 2)
    c.clamp_(min=0.0)
    return c.div_(c.amax((1, 2), keepdim=True))


def _hist(g, *shape):
    w = torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) + 0.2
    return w / w.sum(-1, keepdim=True)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("dense", "unbalanced", "grad"):
        g, dt = _gen(seed), _DT[case["dtype"]]
        s["M"] = _cost(_cloud(g, 1, case["n"], 2), _cloud(g, 1, case["m"], 2))[0].to(dt)
        s["a"], s["b"] = _hist(g, case["n"]).to(dt), _hist(g, case["m"]).to(dt)
        if kind == "unbalanced":
            s["b"] = s["b"] * 1.5
        if kind == "grad":
            for k in ("M", "a", "b"):
                s[k].requires_grad_(True)
    elif kind == "batch":
        g, dt = _gen(seed), _DT[case["dtype"]]
        s["M"] = _cost(_cloud(g, case["B"], case["n"], 2), _cloud(g, case["B"], case["m"], 2)).to(dt)
        s["a"], s["b"] = _hist(g, case["B"], case["n"]).to(dt), _hist(g, case["B"], case["m"]).to(dt)
    elif kind == "ragged":
        # clouds that a data loader hands over: host arrays, one per problem, of the case's sizes
        sizes = np.random.default_rng(case["sizes"]).integers(case["lo"], case["hi"] + 1, (case["B"], 2))
        r = np.random.default_rng(seed)
        s["X"], s["Y"] = [], []
        for n, m in sizes:
            s["X"].append(r.standard_normal((n, case["d"])).astype(np.float32))
            s["Y"].append((0.5 + r.standard_normal((m, case["d"]))).astype(np.float32))
        s["reg"] = np.exp(r.uniform(math.log(case["reg_lo"]), math.log(case["reg_hi"]), case["B"]))
    elif kind == "pairs":
        g = _gen(seed)
        s["X"] = _cloud(g, case["B"], case["n"], case["d"]).float()
        s["Y"] = _cloud(g, case["B"], case["m"], case["d"]).float()
    elif kind == "lazy":
        g = _gen(seed)
        s["X"] = _cloud(g, 1, case["n"], case["d"], 8)[0].float()
        s["Y"] = _cloud(g, 1, case["m"], case["d"], 8)[0].float()
        s["a"], s["b"] = _hist(g, case["n"]).float(), _hist(g, case["m"]).float()
        # regularisation relative to the typical squared distance 2 d (1 + 0.16)
        s["reg"] = case["reg"] * 2.32 * case["d"]
    else:
        g = _gen(seed)
        x, y = _cloud(g, 1, case["n"], 3), _cloud(g, 1, case["m"], 5)
        s["C1"], s["C2"] = _cost(x, x)[0].float(), _cost(y, y)[0].float()
        s["C1"], s["C2"] = 0.5 * (s["C1"] + s["C1"].T), 0.5 * (s["C2"] + s["C2"].T)
        s["p"], s["q"] = _hist(g, case["n"]).float(), _hist(g, case["m"]).float()
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "dense":
        P, lg = pg.sinkhorn(s["a"], s["b"], s["M"], c["reg"], method=c["method"], numItermax=c["iters"],
                            stopThr=c["tol"], log=True, warn=False)
        names = ("u", "v") if c["method"] == "sinkhorn" else ("log_u", "log_v")
        return {"plan": P, "u": lg[names[0]], "v": lg[names[1]]}
    if kind == "unbalanced":
        P, lg = pg.sinkhorn_unbalanced(s["a"], s["b"], s["M"], c["reg"], c["reg_m"], numItermax=c["iters"],
                                       stopThr=c["tol"], log=True)
        return {"plan": P, "u": lg["logu"], "v": lg["logv"]}
    if kind == "grad":
        loss = pg.sinkhorn2(s["a"], s["b"], s["M"], c["reg"], method=c["method"], numItermax=c["iters"],
                            stopThr=c["tol"])
        gM, ga, gb = torch.autograd.grad(loss, (s["M"], s["a"], s["b"]))
        return {"loss": loss.detach(), "gM": gM, "ga": ga, "gb": gb}
    if kind == "batch":
        r = pg.solve_batch(s["M"], c["reg"], s["a"], s["b"], max_iter=c["iters"], tol=c["tol"])
        return {"plan": r.plan, "u": r.potentials[0], "v": r.potentials[1], "value_linear": r.value_linear}
    if kind == "ragged":
        r = pb.solve_sample_ragged(s["X"], s["Y"], s["reg"], reg_relative=True, max_iter=c["iters"], tol=c["tol"])
        return {"u": r.u, "v": r.v}
    if kind == "pairs":
        r = wp.solve_cloud_pairs(s["X"], s["Y"], c["reg"])
        return {"u": r.log_u, "v": r.log_v}
    if kind == "lazy":
        f, g = pg.empirical_sinkhorn(s["X"], s["Y"], s["reg"], s["a"], s["b"], numIterMax=c["iters"], stopThr=0.0,
                                     isLazy=True, warn=False)
        return {"u": f, "v": g}
    T, lg = pg.gromov.entropic_gromov_wasserstein(s["C1"], s["C2"], s["p"], s["q"], epsilon=c["eps"],
                                                  max_iter=c["outer"], tol=1e-9, log=True, numItermax=c["inner"],
                                                  stopThr=0.0, warn=False)
    return {"plan": T, "gw_dist": lg["gw_dist"]}


def work(case):
    kind = case["kind"]
    if kind == "egw":
        n, m, e = case["n"], case["m"], 4
        return {"bytes": e * (n * n + m * m + n * m + n + m),
                "flops": (case["outer"] + 1) * 2.0 * (n * n * m + n * m * m) + case["outer"] * case["inner"] * 4.0 * n * m}
    if kind == "lazy":
        n, m, d = case["n"], case["m"], case["d"]
        return {"bytes": 4.0 * (n + m) * (d + 2), "flops": 2.0 * case["iters"] * n * m * (2 * d + 4)}
    if kind == "pairs":
        # about ten iterations meet the threshold
        B, n, m, d = case["B"], case["n"], case["m"], case["d"]
        return {"bytes": 4.0 * B * (n + m) * (d + 1), "flops": B * n * m * (3.0 * d + 10 * 4.0)}
    if kind == "ragged":
        # sizes are uniform in [lo, hi]; about a hundred iterations meet the threshold
        mid = 0.5 * (case["lo"] + case["hi"])
        return {"bytes": 4.0 * case["B"] * 2 * mid * (case["d"] + 1),
                "flops": case["B"] * mid * mid * (3.0 * case["d"] + 100 * 4.0)}
    e = 8 if case["dtype"] == "f64" else 4
    B, n, m = case.get("B", 1), case["n"], case["m"]
    iters = case["iters"] if case["tol"] == 0.0 else 50  # a few tens of iterations meet the threshold
    # the cost in, the plan (or the gradient of the cost) out
    return {"bytes": float(e * B * (2 * n * m + 4 * (n + m))), "flops": 4.0 * B * n * m * iters}


# ---------------------------------------------------------------------------
# The same results in 64 bits
# ---------------------------------------------------------------------------
def _scaling(K, a, b, u, iters, tol):
    """Scaling iterations v = b / K^T u, u = a / K v of a batch (B, n, m), each
    problem keeping the pair of its first check (every tenth iteration) with a
    column-marginal error below tol, or of the last iteration."""
    Kt = K.transpose(1, 2)
    done = torch.zeros(K.shape[0], dtype=torch.bool, device=K.device)
    U, V = u.clone(), torch.zeros_like(b)
    for it in range(iters):
        v = b / torch.bmm(Kt, u[:, :, None])[:, :, 0]
        u = a / torch.bmm(K, v[:, :, None])[:, :, 0]
        U = torch.where(done[:, None], U, u)
        V = torch.where(done[:, None], V, v)
        if tol > 0.0 and it % 10 == 0:
            err = torch.linalg.vector_norm(v * torch.bmm(Kt, u[:, :, None])[:, :, 0] - b, dim=1)
            done |= err < tol
            if bool(done.all()):
                break
    return U, V


def _exact_dense(case, s):
    M, a, b = (s[k].detach().double() for k in ("M", "a", "b"))
    K = torch.exp(M / -case["reg"])
    log = case["method"] == "sinkhorn_log"
    u0 = torch.full((1, case["n"]), 1.0 if log else 1.0 / case["n"], dtype=torch.float64, device="cuda")
    u, v = (x[0] for x in _scaling(K[None], a[None], b[None], u0, case["iters"], case["tol"]))
    return M, a, b, u, v, K.mul_(u[:, None]).mul_(v[None, :]), log


def exact(case, seed):
    kind = case["kind"]
    if kind == "pairs":
        # an accelerated iteration that stops at a tolerance: its potentials are fixed up to that
        # tolerance and to a constant of its own path only
        return None
    s = prepare(case, seed)
    if kind == "dense":
        _, _, _, u, v, P, log = _exact_dense(case, s)
        return {"plan": P, "u": u.log() if log else u, "v": v.log() if log else v}
    if kind == "grad":
        M, a, b, _, _, P, _ = _exact_dense(case, s)
        n, m = case["n"], case["m"]
        MP = M * P
        # the marginal constraints' implicit derivative, gauge b . mu = 0
        H = torch.zeros(n + m + 1, n + m + 1, dtype=torch.float64, device="cuda")
        H[:n, :n], H[n:n + m, n:n + m] = torch.diag(a), torch.diag(b)
        H[:n, n:n + m], H[n:n + m, :n] = P, P.T
        H[n + m, n:n + m], H[n:n + m, n + m] = b, b
        rhs = torch.cat([MP.sum(1), MP.sum(0), torch.zeros(1, dtype=torch.float64, device="cuda")])
        z = torch.linalg.solve(H, rhs)
        lam, mu = z[:n], z[n:n + m]
        return {"loss": MP.sum(), "gM": P * (1 + (lam[:, None] + mu[None, :] - M) / case["reg"]), "ga": lam, "gb": mu}
    if kind == "unbalanced":
        M, a, b = (s[k].double() for k in ("M", "a", "b"))
        K = torch.exp(M / -case["reg"]) * a[:, None] * b[None, :]
        fi = case["reg_m"] / (case["reg_m"] + case["reg"])
        v = torch.ones_like(b)
        for _ in range(case["iters"]):
            u = (a / (K @ v)) ** fi
            v = (b / (K.T @ u)) ** fi
        return {"plan": u[:, None] * K * v[None, :], "u": torch.log(u + 1e-300), "v": torch.log(v + 1e-300)}
    if kind == "batch":
        # the batched solver updates u first: the same iteration on the transposed problems; it stops as one
        M, a, b = (s[k].double() for k in ("M", "a", "b"))
        K = torch.exp(M / -case["reg"])
        Kt = K.transpose(1, 2)
        v = torch.ones_like(b)
        for it in range(case["iters"]):
            u = a / torch.bmm(K, v[:, :, None])[:, :, 0]
            v = b / torch.bmm(Kt, u[:, :, None])[:, :, 0]
            if it % 10 == 0:
                err = torch.linalg.vector_norm(u * torch.bmm(K, v[:, :, None])[:, :, 0] - a, dim=1)
                if float(err.max()) < case["tol"]:
                    break
        P = u[:, :, None] * K * v[:, None, :]
        return {"plan": P, "u": u.log(), "v": v.log(), "value_linear": (P * M).sum((1, 2))}
    if kind == "ragged":
        B, hi = case["B"], case["hi"]
        K = torch.zeros(B, hi, hi, dtype=torch.float64, device="cuda")
        a, b = (torch.zeros(B, hi, dtype=torch.float64, device="cuda") for _ in range(2))
        for k, (x, y) in enumerate(zip(s["X"], s["Y"])):
            x, y = (torch.as_tensor(z, device="cuda").double() for z in (x, y))
            C = ((x[:, None, :] - y[None, :, :]) ** 2).sum(2)
            K[k, :len(x), :len(y)] = torch.exp(C / (-s["reg"][k] * C.max()))
            a[k, :len(x)], b[k, :len(y)] = 1.0 / len(x), 1.0 / len(y)
        # padded rows and columns have zero mass and keep zero scalings
        ia, ib = a == 0, b == 0
        Kt = K.transpose(1, 2)
        u = torch.ones_like(a)
        done = torch.zeros(B, dtype=torch.bool, device="cuda")
        U, V = u.clone(), torch.zeros_like(b)
        for it in range(case["iters"]):
            v = torch.where(ib, 0.0, b / torch.bmm(Kt, u[:, :, None])[:, :, 0])
            u = torch.where(ia, 0.0, a / torch.bmm(K, v[:, :, None])[:, :, 0])
            U, V = torch.where(done[:, None], U, u), torch.where(done[:, None], V, v)
            if it % 10 == 0:
                err = torch.linalg.vector_norm(v * torch.bmm(Kt, u[:, :, None])[:, :, 0] - b, dim=1)
                done |= err < case["tol"]
                if bool(done.all()):
                    break
        return {"u": U[~ia].log(), "v": V[~ib].log()}
    if kind == "lazy":
        x, y = s["X"].double(), s["Y"].double()
        C = (x * x).sum(1)[:, None] + (y * y).sum(1)[None, :] - 2.0 * x @ y.T
        K = torch.exp(C.clamp_(min=0.0).div_(-s["reg"]))
        a, b = s["a"].double(), s["b"].double()
        v = torch.ones_like(b)
        for _ in range(case["iters"]):
            # the lazy solver updates f first, from g = 0
            u = a / (K @ v)
            v = b / (K.T @ u)
        return {"u": u.log(), "v": v.log()}
    C1, C2, p, q = (s[k].double() for k in ("C1", "C2", "p", "q"))
    const = ((C1 * C1) @ p)[:, None] + ((C2 * C2) @ q)[None, :]
    T = p[:, None] * q[None, :]
    for _ in range(case["outer"]):
        K = torch.exp((2.0 * const - 4.0 * C1 @ T @ C2) / -case["eps"])
        u = torch.full_like(p, 1.0 / case["n"])
        for _ in range(case["inner"]):
            v = q / (K.T @ u)
            u = p / (K @ v)
        T = u[:, None] * K * v[None, :]
    return {"plan": T, "gw_dist": ((const - 2.0 * C1 @ T @ C2) * T).sum()}
