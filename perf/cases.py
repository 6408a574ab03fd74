"""Performance cases of the sampler: the calls a user's program makes, over the sizes it makes them at.

Models follow the benchmark's law (achr.cu_gb300/synthetic.py): every reaction touches 2-6 metabolites
with coefficients from {-2, -1, 1, 2}, a quarter to a third of the reactions is irreversible, a few are
exchange reactions with tight bounds.  The benchmark finds an interior point with one LP; here the point
comes first (the null-space projection of a random vector) and the bounds are laid around it: columns
whose flux is negative are written in the other direction before they are made irreversible, with at
least one unit of slack, and exchange reactions are taken among the small fluxes.  Warmup points are the
ends of random chords through that point, shrunk toward their mean as the reference's generator does,
either exact or rounded to six decimals as the reference's CSV holds them ("percent_f": every residual
check of the sampler then reprojects).
"""
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()

DEV = "cuda"
KEEP_ABOVE = 4000  # reactions: above this the context takes seconds to build, and a program keeps it


def listed():
    return [
        # The smallest call: a few chains of the E. coli core size (a notebook, a test, a pilot): latency.
        {"name": "small pilot", "call": "sample_device", "m": 72, "n": 95, "chains": 64, "steps": 50,
         "form": "exact", "pool": 0},
        # The reference's published table, second row: E. coli core size, one file of 5000 points from a %f warmup
        # CSV, points back on the host as the command line writes them.  (Runs on %f warmups are cut to 50-100
        # steps: a real run is more of the same, and later steps multiply a last-digit difference.)
        {"name": "small file", "call": "sample", "m": 72, "n": 95, "chains": 5000, "steps": 100,
         "form": "percent_f"},
        # The table's fifth row: the P. putida model's size, 5000 points, host buffers.
        {"name": "mid file", "call": "sample", "m": 911, "n": 1060, "chains": 5000, "steps": 50,
         "form": "percent_f"},
        # The drop-in workload at genome scale: %f warmups, batched reprojection at every check.
        {"name": "genome percent_f", "call": "sample_device", "m": 2766, "n": 3742, "chains": 8000, "steps": 50,
         "form": "percent_f", "pool": 0},
        # Checkpointed sampling at genome scale (ESS traces, long runs cut into segments): plain chain kernel.
        {"name": "genome segments", "call": "sample_resume", "m": 2766, "n": 3742, "chains": 3000, "steps": 100,
         "form": "exact"},
        # Hit-and-run along a learned direction pool at genome scale.
        {"name": "genome directions", "call": "sample_device", "m": 2766, "n": 3742, "chains": 3000, "steps": 100,
         "form": "exact", "pool": 4096},
        # Many models of uneven size in one launch.
        {"name": "model batch", "call": "sample_batch", "models": 8, "lo": 95, "hi": 1500, "chains": 6000,
         "steps": 100, "form": "exact"},
        # The largest model: sampling with a periodic batched reprojection.
        {"name": "large periodic", "call": "sample_periodic", "m": 5063, "n": 7440, "chains": 2000, "steps": 100,
         "period": 50, "form": "exact"},
        # One batched reprojection of a block of chains of the largest model.
        {"name": "large reprojection", "call": "reproject", "m": 5063, "n": 7440, "chains": 16384, "rounds": 2},
        # One forward and backward pass of the direction preconditioner, genome-scale basis and rank.
        {"name": "genome loss and gradient", "call": "loss_grad", "d": 940, "r": 256, "batch": 4096},
        # The same for the small model's basis: launches and latency.
        {"name": "small loss and gradient", "call": "loss_grad", "d": 9, "r": 4, "batch": 4096},
        # Null-space coordinates of a block of samples (the preconditioner's training set).
        {"name": "genome coordinates", "call": "null_coords", "m": 2766, "n": 3742, "chains": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["sample_device", "sample", "sample_device", "sample_resume", "directions", "sample_batch",
                       "sample_periodic", "reproject", "loss_grad", "loss_grad", "null_coords"])
    if call == "loss_grad":
        r = _log(rng, 4, 256)
        d = _log(rng, r + 5, 2358)
        return {"call": call, "d": d, "r": r, "batch": min(_log(rng, 512, 8192), 940 * 4096 // d + 512)}
    if call == "sample_batch":
        return {"call": call, "models": rng.randint(2, 8), "lo": 95, "hi": _log(rng, 300, 1500),
                "chains": _log(rng, 300, 6000), "steps": rng.randint(20, 100), "form": "exact"}
    n = _log(rng, 95, 3742)
    case = {"call": call, "m": int(n * rng.uniform(0.68, 0.86)), "n": n}
    if call in ("reproject", "null_coords"):
        case["chains"] = _log(rng, 100, 16384)
        if call == "reproject":
            case["rounds"] = rng.randint(1, 3)
        return case
    form = rng.choice(["exact", "percent_f"]) if call in ("sample", "sample_device") else "exact"
    case["steps"] = rng.randint(11, 60 if form == "percent_f" else 120)
    # chain-steps x reactions up to the genome cases', as many chains as a user of that size runs
    case["chains"] = max(1, min(_log(rng, 50, 8000), int(1.0e9 / (n * case["steps"]))))
    if call == "directions":
        return {**case, "call": "sample_device", "form": "exact", "pool": _log(rng, 200, 4096)}
    if call == "sample_periodic":
        return {**case, "period": rng.randint(10, 60), "form": "exact"}
    case["form"] = form
    if call == "sample_device":
        case["pool"] = 0
    return case


# --- models and warmup points ------------------------------------------------------------------------------

_models = {}   # (m, n) -> model arrays, dense S, null-space basis, interior point
_handles = {}  # (m, n, form) -> (sampler, warmup points) of the sizes whose context a program keeps


class _M:
    pass


def _model(m, n):
    if (m, n) in _models:
        return _models[(m, n)]
    rng = np.random.default_rng(1000003 * m + n)
    rows, cols, vals = [], [], []
    for j in range(n):
        k = min(int(rng.integers(2, 7)), m)
        mets = np.sort(rng.choice(m, size=k, replace=False))
        rows.append(mets)
        cols.append(np.full(k, j))
        vals.append(np.array([-2.0, -1.0, 1.0, 2.0])[rng.integers(0, 4, k)])
    row, col, val = (np.concatenate(v) for v in (rows, cols, vals))
    S = torch.zeros((m, n), dtype=torch.float64, device=DEV)
    S[torch.from_numpy(row).to(DEV), torch.from_numpy(col).to(DEV)] = torch.from_numpy(val).to(DEV)
    lam, V = torch.linalg.eigh(S.T @ S)
    N = V[:, lam.abs() < n * lam.abs().max() * 2.2204e-16].contiguous()
    del lam, V
    N[N.norm(dim=1) < 1e-9] = 0.0  # reactions no flux passes through
    v0 = 30.0 * (N @ (N.T @ torch.from_numpy(rng.standard_normal(n)).to(DEV)))
    flip = torch.where(v0 < 0, -1.0, 1.0).to(torch.float64)
    S *= flip
    N *= flip[:, None]
    v0 = v0.abs()
    val = val * flip.cpu().numpy()[col]
    v = v0.cpu().numpy()
    lb, ub = np.full(n, -1000.0), np.full(n, 1000.0)
    order = rng.permutation(n)
    n_ex = max(2, n // 25)
    ex = [i for i in order if 0 < v[i] < 10.0][:n_ex]
    lb[ex], ub[ex] = -20.0, 20.0
    rest = [i for i in order if (v[i] >= 1.0 or v[i] == 0.0) and lb[i] < -100.0]
    lb[rest[: int(0.3 * n)]] = 0.0
    M = _M()
    M.m, M.n, M.S, M.N, M.v0 = m, n, S, N, v0
    M.lb, M.ub = (torch.from_numpy(b).to(DEV) for b in (lb, ub))
    M.host = pkg.HostModel(n, m, row.astype(np.int32), col.astype(np.int32), val, lb, ub)
    M.nnz = len(val)
    _models[(m, n)] = M
    return M


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _chords(M, count, g):
    """(count, n) points where random chords through the interior point leave the box, far and near ends in turn."""
    out = torch.empty((count, M.n), dtype=torch.float64, device=DEV)
    up, lo = M.ub - M.v0, M.lb - M.v0
    for j in range(0, count, 2048):
        k = min(2048, count - j)
        D = torch.randn((k, M.N.shape[1]), dtype=torch.float64, device=DEV, generator=g) @ M.N.T
        t = torch.where(D > 0, up / D, torch.where(D < 0, lo / D, math.inf)).amin(1)
        u = torch.where(D > 0, lo / D, torch.where(D < 0, up / D, -math.inf)).amax(1)
        far = (torch.arange(j, j + k, device=DEV) % 2 == 1)
        out[j:j + k] = M.v0 + torch.where(far, t, u)[:, None] * D
    return torch.minimum(torch.maximum(out, M.lb), M.ub)


def _warmup(M, seed, form):
    """(2n, n): row j is warmup point j (the sampler's column j)."""
    w = _chords(M, 2 * M.n, _gen(seed))
    w = 0.33 * w + 0.67 * w.mean(0)
    return torch.round(w * 1e6) / 1e6 if form == "percent_f" else w


def _sampler(case, seed, form):
    """(sampler, its warmup points): a new context for the seed's warmup points, or the kept one of a large model."""
    M = _model(case["m"], case["n"])
    kept = M.n > KEEP_ABOVE
    key = (M.m, M.n, form)
    if kept and key in _handles:
        return _handles[key]
    w = _warmup(M, 7 if kept else seed, form)
    got = pkg.Sampler(M.host, w.cpu().numpy().T), w
    if kept:
        _handles[key] = got
    return got


def _batch(case):
    """(m, n, chains) of every model of a batch: sizes log-uniform, chains in proportion to the size."""
    k = case["models"]
    ns = [int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / k))) for i in range(k)]
    return [(int(round(0.7 * n)), n, max(1, case["chains"] * n // sum(ns))) for n in ns]


def _points(M, count, seed):
    """(n, count) points off the null space by 1e-6 in the row space of S, as sampling on %f warmups leaves them."""
    g = _gen(seed + 5)
    x = 0.33 * _chords(M, count, g) + 0.67 * M.v0
    x += 1e-6 * torch.randn((count, M.m), dtype=torch.float64, device=DEV, generator=g) @ M.S
    return torch.minimum(torch.maximum(x, M.lb), M.ub).T.contiguous()


def _precond(case, seed):
    """Parameters part of the way to those of the samples they are fitted to, in coordinates of unit spread."""
    d, r, B = case["d"], case["r"], case["batch"]
    g = _gen(seed)
    rand = lambda *shape: torch.randn(shape, device=DEV, generator=g)  # noqa: E731
    s, U = 0.3 * rand(d), 0.8 * rand(d, r) / math.sqrt(r)
    Y = torch.exp(s + 0.3 * rand(d))[:, None] * rand(d, B) + (0.5 * U + 0.4 * rand(d, r) / math.sqrt(r)) @ rand(r, B)
    return s, U.contiguous(), Y.contiguous()


def prepare(case, seed):
    st = {"case": case, "seed": seed}
    call = case["call"]
    f64 = {"dtype": torch.float64, "device": DEV}
    if call == "loss_grad":
        st["s"], st["U"], st["Y"] = _precond(case, seed)
        st["gs"], st["gU"] = torch.empty_like(st["s"]), torch.empty_like(st["U"])
        return st
    if call == "sample_batch":
        st["samplers"], st["out"] = [], []
        for k, (m, n, p) in enumerate(_batch(case)):
            st["samplers"].append(_sampler({"m": m, "n": n}, seed + k, case["form"])[0])
            st["out"].append(torch.empty((n, p), **f64))
        return st
    st["smp"], w = _sampler(case, seed, case.get("form", "exact"))
    n, P = case["n"], case["chains"]
    if call == "sample":
        return st
    st["x"] = torch.empty((n, P), **f64)
    if call in ("sample_resume", "sample_periodic"):
        st["A"] = torch.empty((n, P), **f64)
    if call == "reproject":
        st["x0"] = _points(_model(case["m"], n), P, seed)
    if call == "null_coords":
        st["x"] = _points(_model(case["m"], n), P, seed)
        st["mu"] = w.mean(0)
        st["Y"] = torch.empty((st["smp"].precond_dim()[0], P), device=DEV)
    if case.get("pool"):
        D = _pool(case, seed)
        st["smp"].set_directions(d_dirs=D.data_ptr(), ld=n, n_dirs=case["pool"])
    return st


def _pool(case, seed):
    M = _model(case["m"], case["n"])
    return torch.randn((case["pool"], M.N.shape[1]), dtype=torch.float64, device=DEV, generator=_gen(seed + 3)) @ M.N.T


def run(st):
    case, seed = st["case"], st["seed"]
    call = case["call"]
    if call == "loss_grad":
        loss = pkg.precond_loss_grad(case["d"], case["r"], case["batch"], st["s"].data_ptr(), st["U"].data_ptr(),
                                     st["Y"].data_ptr(), case["batch"], st["gs"].data_ptr(), st["gU"].data_ptr())
        return {"loss": loss, "gs": st["gs"], "gU": st["gU"]}
    if call == "sample_batch":
        out = st["out"]
        pkg.sample_batch(st["samplers"], [o.shape[1] for o in out], case["steps"], [o.data_ptr() for o in out],
                         [o.shape[1] for o in out], seed=seed)
        return out
    smp, P = st["smp"], case["chains"]
    if call == "sample":
        pts, stats = smp.sample(P, case["steps"], seed=seed)
        return {"points": pts, **{k: stats[k] for k in ("accepted", "rejected", "checks", "reprojections")}}
    x = st["x"]
    if call == "sample_device":
        smp.sample_device(P, case["steps"], x.data_ptr(), P, seed=seed)
        return x
    if call == "sample_resume":
        half = case["steps"] // 2
        smp.sample_resume(P, 0, half, False, x.data_ptr(), st["A"].data_ptr(), P, seed=seed)
        smp.sample_resume(P, half, case["steps"] - half, True, x.data_ptr(), st["A"].data_ptr(), P, seed=seed)
        return {"x": x, "A": st["A"]}
    if call == "sample_periodic":
        smp.sample_periodic(P, case["steps"], case["period"], x.data_ptr(), st["A"].data_ptr(), P, seed=seed)
        return {"x": x, "A": st["A"]}
    if call == "reproject":
        x.copy_(st["x0"])
        smp.reproject(P, x.data_ptr(), P, max_rounds=case["rounds"], with_stats=False)
        return x
    smp.null_coords(P, x.data_ptr(), P, st["Y"].data_ptr(), P, d_mu=st["mu"].data_ptr())
    return st["Y"]


def work(case):
    call = case["call"]
    if call == "loss_grad":
        d, r, B = case["d"], case["r"], case["batch"]
        # W^T Y, Minv Q, W Rq, V^T U, V T; M, its inverse, W Minv
        return {"bytes": 4.0 * (d * B + 2 * d * r + 2 * d), "flops": 2.0 * (4 * d * r * B + r * r * B + 2 * d * r * r + r ** 3)}
    if call == "sample_batch":
        parts = [work({"call": "sample_device", "m": m, "n": n, "chains": p, "steps": case["steps"],
                       "form": case["form"], "pool": 0}) for m, n, p in _batch(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    m, n, P = case["m"], case["n"], case["chains"]
    if call == "null_coords":
        d = n - m
        return {"bytes": 8.0 * n * (P + d) + 4.0 * d * P, "flops": 2.0 * n * d * P}
    project = 2.0 * 8 * n * P, 2.0 * m * m * P + 16.0 * n * P  # x read and written, S x, (S S^T)^+ r, S^T z
    if call == "reproject":
        return {"bytes": project[0] + 4.0 * m * m, "flops": project[1]}
    # a step: w - c, two bound distances and ratios, x + t u, the centre; S x (4 entries a column) every 10th
    steps = P * case["steps"]
    got = {"bytes": 8.0 * n * (case.get("pool") or 2 * n) + 8.0 * n * P, "flops": (11.0 + 0.8) * n * steps}
    if call in ("sample_resume", "sample_periodic"):
        got["bytes"] += 8.0 * n * P
    if case["form"] == "percent_f":
        got["flops"] += project[1] * (case["steps"] + 9) // 10
    return got


# --- the same calls in 64 bits, by plain torch and numpy -----------------------------------------------------

def _philox(step, attempt, chain, seed):
    """Philox4x32-10 words of (step, attempt, chain) under key seed, for an array of chain ids."""
    u = lambda v: np.asarray(v, dtype=np.uint64)  # noqa: E731
    mask = u(0xFFFFFFFF)
    c0, c1 = np.full(chain.shape, step, np.uint64), np.full(chain.shape, attempt, np.uint64)
    c2, c3 = chain & mask, chain >> u(32)
    k0, k1 = int(seed) & 0xFFFFFFFF, int(seed) >> 32
    for _ in range(10):
        p0, p1 = u(0xD2511F53) * c0, u(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> u(32)) ^ c1 ^ u(k0), p1 & mask, (p0 >> u(32)) ^ c3 ^ u(k1), p0 & mask
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c2, c3


def _project(M, X):
    """Rows of X onto the null space of S."""
    return (X @ M.N) @ M.N.T


def _walk(M, cols, centre, seed, first, P, steps, pool=False, period=0):
    """(points, centre accumulators), each (n, P), of chains first .. first + P - 1 (the reference's step, all chains at once)."""
    W = cols.shape[0]
    chain = np.arange(first, first + P, dtype=np.uint64)
    X, A = centre.repeat(P, 1), (0.0 if pool else float(W)) * centre.repeat(P, 1)
    Ssp = M.S.to_sparse()
    for s in range(steps):
        todo = np.arange(P)
        _, w2, w3 = _philox(s, 0, chain, seed)
        U = torch.from_numpy(((((w2 << np.uint64(32)) | w3) >> np.uint64(12)).astype(np.float64) + 0.5) * 2.0 ** -52)
        U = U.to(DEV)
        new = X.clone()
        for att in range(1000):
            w0 = _philox(s, att, chain[todo], seed)[0]
            t = torch.from_numpy(todo).to(DEV)
            u = cols[torch.from_numpy(((w0 * np.uint64(W)) >> np.uint64(32)).astype(np.int64)).to(DEV)]
            if not pool:
                u = u - A[t] / float(W + s)
            u = u / u.norm(dim=1, keepdim=True)
            up, dn = M.ub - X[t], X[t] - M.lb
            on = (up > 1e-14) & (dn > 1e-14) & (u.abs() > 1e-9)
            hi = torch.where(on, torch.where(u > 0, up, dn) / u.abs(), math.inf).amin(1)
            lo = torch.where(on, torch.where(u > 0, dn, up) / u.abs(), math.inf).amin(1)
            ok = on.any(1) & ~((hi < 1e-9) & (lo < 1e-9))
            step = U[t] * (hi + lo) - lo
            new[t[ok]] = X[t[ok]] + step[ok, None] * u[ok]
            todo = todo[~ok.cpu().numpy()]
            if not len(todo):
                break
        if s % 10 == 0:
            far = (Ssp @ new.T).abs().amax(0) > 1e-9
            if far.any():
                new[far] = _project(M, new[far])
        X = torch.minimum(torch.maximum(new, M.lb), M.ub)
        if not pool:
            A = A + X
        if period and ((s + 1) % period == 0 or s + 1 == steps) and (Ssp @ X.T).abs().max() > 1e-9:
            Y = torch.minimum(torch.maximum(_project(M, X), M.lb), M.ub)
            A, X = A + (Y - X), Y
    return X.T.contiguous(), A.T.contiguous()


def exact(case, seed):
    call = case["call"]
    if call == "loss_grad":
        s, U, Y = (t.double() for t in _precond(case, seed))
        a, B = torch.exp(-2.0 * s), case["batch"]
        W = a[:, None] * U
        R = torch.eye(case["r"], dtype=torch.float64, device=DEV) + U.T @ W
        Minv = torch.linalg.inv(R)
        V = a[:, None] * Y - W @ (Minv @ (W.T @ Y))
        K = W @ Minv
        loss = 0.5 * ((Y * V).sum() / B + 2.0 * s.sum() + torch.logdet(R))
        gs = torch.exp(2.0 * s) * (a - (K * W).sum(1) - (V * V).sum(1) / B)
        return {"loss": float(loss), "gs": gs, "gU": K - V @ (V.T @ U) / B}
    if call == "null_coords":
        return None  # the basis is the framework's own choice
    if call == "sample_batch":
        out, first = [], 0
        for k, (m, n, p) in enumerate(_batch(case)):
            M = _model(m, n)
            w = _warmup(M, seed + k, case["form"])
            out.append(_walk(M, w, w.mean(0), seed, first, p, case["steps"])[0])
            first += p
        return out
    M = _model(case["m"], case["n"])
    P = case["chains"]
    if call == "reproject":
        x = _points(M, P, seed)
        return torch.minimum(torch.maximum(_project(M, x.T), M.lb), M.ub).T.contiguous()
    w = _warmup(M, 7 if M.n > KEEP_ABOVE else seed, case["form"])
    cols = _pool(case, seed) if case.get("pool") else w
    x, A = _walk(M, cols, w.mean(0), seed, 0, P, case["steps"], bool(case.get("pool")), case.get("period", 0))
    if call == "sample":
        return {"points": x}
    return x if call == "sample_device" else {"x": x, "A": A}
