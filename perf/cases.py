"""Performance cases of polar_b200: the work a user has it do, through its public entry points.

Kinds of case (the fields of each are listed in `listed` and `draw`):

* apply     `pg.Op(G)(x)`: one operator product y = (L + sigma I) x.
* solve     `pg.msolve`: one multi-shift CG solve on the poles of x^-s, its iterates kept on
            the endpoints of a candidate pool.  FP64 solves track the solution norms, as the
            greedy's shortlist solves and the certified marginals do; mixed-precision solves do
            not, as the bank.  `added` weighted edges on the operator make it one block of the
            relaxed-weight adjoint.
* batch     `polar_b200.batch.msolve_batch`: one solve per graph over several graphs.
* score     `polar_score_topb` (C ABI): proxy scores of all candidates and the stable top-B.
* maintain  `polar_maintain` (C ABI): Sherman-Morrison update of the banks and caches.
* greedy    `pg.polar`: a whole greedy from given sketches.

Graphs are seeded Chung-Lu graphs with the vertex counts, mean degrees and exponents of
`polar_b200.synth.CONFIGS`, drawn on the GPU.  FP64 solves run to 1e-10, the default of the
certified marginals and of the relaxed gradient; mixed ones to the workloads' 1e-6 and 1e-7.
"""
import math

import numpy as np
import torch

import polar_b200 as pg
from polar_b200 import _lib
from polar_b200.batch import msolve_batch
from polar_b200.solver import prepare_active

DEV = "cuda"


def listed():
    return [
        # the smallest call: one vector through the operator of the plain workload's graph
        dict(name="apply-n2000-r1-f64", kind="apply", n=2000, deg=6.0, gamma=2.5, R=1, prec="fp64", weighted=False),
        # an odd block width on the com-DBLP-sized graph (residual check of a 20-column solve)
        dict(name="apply-n317k-r20-f64", kind="apply", n=317080, deg=6.62, gamma=2.4, R=20, prec="fp64",
             weighted=False),
        # one certified marginal: a single incidence column, two active rows, the plain workload
        dict(name="solve-n2000-r1-f64", kind="solve", n=2000, deg=6.0, gamma=2.5, R=1, K=16, rows=2,
             sigma=1e-2, cols="edge", prec="fp64", tol=1e-10, added=0, weighted=False),
        # the shortlist solve of a 20,000-vertex graph
        dict(name="solve-n20k-r16-f64", kind="solve", n=20000, deg=6.62, gamma=2.4, R=16, K=24, rows=17200,
             sigma=1e-2, cols="edge", prec="fp64", tol=1e-10, added=0, weighted=False),
        # the shortlist solve of the com-DBLP-sized workload in FP64
        dict(name="solve-n317k-r16-f64", kind="solve", n=317080, deg=6.62, gamma=2.4, R=16, K=24, rows=227000,
             sigma=1e-2, cols="edge", prec="fp64", tol=1e-10, added=0, weighted=False),
        # its bank: the 2q = 128 sketch columns in mixed precision
        dict(name="bank-n317k-r128-mixed", kind="solve", n=317080, deg=6.62, gamma=2.4, R=128, K=24,
             rows=227000, sigma=1e-2, cols="sketch", prec="mixed", tol=1e-7, added=0, weighted=False),
        # the com-LiveJournal-sized workload: 16 incidence columns over the endpoints of a million
        # candidates
        dict(name="solve-n4M-r16-mixed", kind="solve", n=3997962, deg=17.35, gamma=2.1, R=16, K=32,
             rows=1574065, sigma=1e-1, cols="edge", prec="mixed", tol=1e-6, added=0, weighted=False),
        # one 64-column block of the relaxed-weight adjoint: 4,096 weighted edges on the operator
        dict(name="adjoint-n50k-r64-f64", kind="solve", n=50000, deg=5.27, gamma=2.2, R=64, K=24, rows=7500,
             sigma=1e-1, cols="edge", prec="fp64", tol=1e-10, added=4096, weighted=False),
        # a study over many graphs: eight banks of 64 columns in one call
        dict(name="batch-8-r64-mixed", kind="batch", graphs=8, nmin=5000, nmax=60000, R=64, K=16, rows=4000,
             prec="mixed", tol=1e-7),
        # scoring a million candidates over 32 poles and taking the 16 best
        dict(name="score-n1M-p32-b16", kind="score", N=1000000, p=32, B=16, obj=0, all=False),
        # one round's maintenance of the com-DBLP-sized banks in mixed precision
        dict(name="maintain-n317k-q64-mixed", kind="maintain", rows=226000, N=200000, p=24, q=64, B=16, prec="mixed"),
        # a whole greedy on the plain workload's graph
        dict(name="greedy-n2000-k4", kind="greedy", n=2000, deg=6.0, gamma=2.5, N=20000, K=16, q=32, B=4, k=4,
             tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "solve", "solve", "solve", "solve", "adjoint", "batch", "score", "maintain",
                       "greedy"])
    deg = round(rng.uniform(4.0, 18.0), 2)
    gamma = round(rng.uniform(2.1, 2.6), 2)
    if kind == "apply":
        prec = rng.choice(["fp64", "mixed"])
        R = rng.choice([1, rng.randint(2, 32), 16, 64])
        return dict(kind="apply", n=_log_int(rng, 1500, 1200000), deg=deg, gamma=gamma, R=R, prec=prec,
                    weighted=rng.random() < 0.25)
    if kind == "solve":
        prec = rng.choice(["fp64", "mixed"])
        n = _log_int(rng, 1500, 320000)
        R = rng.choice([1, rng.randint(2, 16), 16, 64 if prec == "fp64" else 128])
        return dict(kind="solve", n=n, deg=deg, gamma=gamma, R=R, K=rng.randint(8, 32),
                    rows=2 if R == 1 else _log_int(rng, 500, n * 7 // 10), sigma=rng.choice([1e-2, 1e-1]),
                    cols="sketch" if R > 16 else "edge", prec=prec, tol=1e-10 if prec == "fp64" else rng.choice([1e-6, 1e-7]), added=0,
                    weighted=rng.random() < 0.2)
    if kind == "adjoint":
        return dict(kind="solve", n=_log_int(rng, 5000, 60000), deg=deg, gamma=gamma, R=rng.randint(17, 64),
                    K=rng.randint(8, 24), rows=_log_int(rng, 500, 4000), sigma=1e-1, cols="edge", prec="fp64",
                    tol=1e-10, added=_log_int(rng, 16, 4096), weighted=False)
    if kind == "batch":
        return dict(kind="batch", graphs=rng.randint(2, 8), nmin=5000, nmax=_log_int(rng, 10000, 60000),
                    R=rng.randint(33, 64), K=rng.randint(8, 16), rows=_log_int(rng, 500, 4500), prec="mixed",
                    tol=1e-7)
    if kind == "score":
        return dict(kind="score", N=_log_int(rng, 5000, 1000000), p=rng.randint(8, 32), B=rng.randint(1, 32),
                    obj=rng.choice([0, 0, 2]), all=rng.random() < 0.5)
    if kind == "maintain":
        return dict(kind="maintain", rows=_log_int(rng, 3000, 226000), N=_log_int(rng, 3000, 200000),
                    p=rng.randint(8, 24), q=rng.choice([32, 64, rng.randint(20, 64)]), B=rng.randint(1, 16),
                    prec=rng.choice(["fp64", "mixed"]))
    return dict(kind="greedy", n=rng.randint(1000, 3000), deg=deg, gamma=2.5, N=rng.randint(3000, 20000),
                K=rng.randint(8, 16), q=rng.choice([16, 32]), B=rng.randint(1, 8), k=rng.randint(2, 4), tol=1e-10)


# ---- inputs ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rand(gen, *shape):
    return torch.rand(shape, dtype=torch.float64, device=DEV, generator=gen)


def _chung_lu(n, mean_deg, gamma, gen):
    """Edges (int64 [m, 2], u < v, sorted) of a Chung-Lu graph: expected degrees
    proportional to (i + i0)^(-1/(gamma - 1)) with the largest at the structural cutoff (at
    most 15,000), no isolated vertices."""
    alpha = 1.0 / (gamma - 1.0)
    i = torch.arange(n, dtype=torch.float64, device=DEV)
    total = n * mean_deg
    dmax = min(15000.0, math.sqrt(total))
    lo, hi = 1e-6, float(n)
    for _ in range(40):
        mid = math.sqrt(lo * hi)
        b = (i + mid) ** (-alpha)
        if total * float(b[0] / b.sum()) > dmax:
            lo = mid
        else:
            hi = mid
    w = (i + hi) ** (-alpha)
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()

    def ends(count):
        return torch.searchsorted(cdf, _rand(gen, count)).clamp_(max=n - 1)

    target = int(round(total / 2))
    draws = int(target * 1.1) + 64
    u, v = ends(draws), ends(draws)
    a, b = torch.minimum(u, v), torch.maximum(u, v)
    keys = torch.unique((a * n + b)[a != b])
    if keys.numel() > target:
        keys = keys[torch.randperm(keys.numel(), device=DEV, generator=gen)[:target]]
    iso = torch.nonzero(torch.bincount(torch.cat([keys // n, keys % n]), minlength=n) == 0).flatten()
    part = ends(iso.numel())
    part = torch.where(part == iso, (iso + 1) % n, part)
    keys = torch.unique(torch.cat([keys, torch.minimum(iso, part) * n + torch.maximum(iso, part)]))
    return torch.stack([keys // n, keys % n], 1)


def _candidates(n, edges, N, gen):
    """N distinct non-edges (int64 [N, 2], u < v) in random order."""
    keys = edges[:, 0] * n + edges[:, 1]
    k = 2 * N + 64
    u = torch.randint(n, (k,), device=DEV, generator=gen)
    v = torch.randint(n, (k,), device=DEV, generator=gen)
    key = torch.unique((torch.minimum(u, v) * n + torch.maximum(u, v))[u != v])
    pos = torch.searchsorted(keys, key).clamp_(max=keys.numel() - 1)
    key = key[keys[pos] != key]
    key = key[torch.randperm(key.numel(), device=DEV, generator=gen)[:N]]
    return torch.stack([key // n, key % n], 1)


def _poles(s, K, sigma, lam):
    """K poles of x^-s: the Gauss-Jacobi rule of t = c (1 - y)/(1 + y), c = sqrt(sigma lam)."""
    i = np.arange(K, dtype=np.float64)
    diag = (1.0 - 2.0 * s) / (4.0 * i ** 2 - 1.0)
    j = np.arange(1, K, dtype=np.float64)
    off = np.sqrt((j - s) * (j + s - 1.0)) / (2.0 * j - 1.0)
    off[:1] *= math.sqrt(2.0)
    y, vec = np.linalg.eigh(np.diag(diag) + np.diag(off, 1) + np.diag(off, -1))
    c = math.sqrt(sigma * lam)
    tau = c * (1.0 - y) / (1.0 + y)
    om = c ** (1.0 - s) * 2.0 * vec[0] ** 2 / (1.0 + y)
    return tau[::-1].copy(), om[::-1].copy()


def _graph_input(c, gen):
    """Edges (device), weights (device or None) and the weighted degrees."""
    E = _chung_lu(c["n"], c["deg"], c["gamma"], gen)
    w = 0.5 + _rand(gen, E.shape[0]) if c.get("weighted") else None
    ww = torch.ones(E.shape[0], dtype=torch.float64, device=DEV) if w is None else w
    deg = torch.zeros(c["n"], dtype=torch.float64, device=DEV)
    deg.index_add_(0, E[:, 0], ww).index_add_(0, E[:, 1], ww)
    return E, w, deg


def _solve_input(c, seed):
    """Everything a solve is given, as plain tensors and arrays."""
    gen = _gen(seed)
    n, R = c["n"], c["R"]
    E, w, deg = _graph_input(c, gen)
    cand = _candidates(n, E, max(R, c["added"]), gen)
    tau, _ = _poles(0.5, c["K"], c["sigma"], c["sigma"] + 2.0 * float(deg.max()) + 40.0)
    # active rows: the columns' own endpoints and those of the rest of the pool
    place = _rand(gen, n)
    if c["cols"] == "edge":
        place[cand[:R].flatten()] = -1.0
    active = torch.sort(torch.argsort(place)[:c["rows"]]).values
    W = torch.zeros((n, R), dtype=torch.float64, device=DEV)
    if c["cols"] == "sketch":
        W.normal_(generator=gen).mul_(1.0 / math.sqrt(R))
        W -= W.mean(0)
    else:  # incidence columns e_a - e_b
        cols = torch.arange(R, device=DEV)
        W[cand[:R, 0], cols] = 1.0
        W[cand[:R, 1], cols] = -1.0
    return dict(E=E, w=w, deg=deg, tau=tau, active=active, W=W, extra=cand[:c["added"]], wx=_rand(gen, c["added"]))


def _graph(c, E, w, sigma):
    return pg.Graph(c["n"], E.cpu().numpy(), sigma, weights=None if w is None else w.cpu().numpy())


def _batch_cases(c):
    """The single-graph solves of a batch: sizes over [nmin, nmax], each with its own sigma."""
    out = []
    for b in range(c["graphs"]):
        f = b / max(1, c["graphs"] - 1)
        n = int(c["nmin"] * (c["nmax"] / c["nmin"]) ** f)
        out.append(dict(kind="solve", n=n, deg=4.0 + (5 * b) % 16, gamma=2.2 + 0.1 * (b % 5), R=c["R"], K=c["K"],
                        rows=c["rows"], sigma=(1e-2, 1e-1)[b % 2], cols="sketch", prec=c["prec"], tol=c["tol"], added=0, weighted=False))
    return out


def _score_input(c, seed):
    gen = _gen(seed)
    p, N = c["p"], c["N"]
    tau, om = _poles(0.5, p, 1e-2, 2000.0)
    tau, om = torch.as_tensor(tau, device=DEV), torch.as_tensor(om, device=DEV)
    # caches of a candidate fall with the pole as those of a resolvent do
    size = torch.exp(0.8 * torch.randn((1, N), dtype=torch.float64, device=DEV, generator=gen))
    t = size / (0.3 + tau[:, None]) * (0.9 + 0.2 * _rand(gen, p, N))
    h = size / (0.3 + tau[:, None]) ** 2 * (0.9 + 0.2 * _rand(gen, p, N))
    live = (_rand(gen, N) > 0.001).to(torch.uint8)
    return dict(h=h, t=t, tau=tau, om=om, live=live)


def _maintain_input(c, seed):
    gen = _gen(seed)
    p, nA, q, N, B = c["p"], c["rows"], c["q"], c["N"], c["B"]
    dt = torch.float32 if c["prec"] == "mixed" else torch.float64
    XY = torch.empty((p, nA, 2 * q), dtype=dt, device=DEV).normal_(generator=gen).mul_(0.3)
    U = torch.empty((p, nA, B), dtype=dt, device=DEV).normal_(generator=gen).mul_(0.01)
    es = torch.randint(nA, (N, 2), device=DEV, generator=gen, dtype=torch.int32)
    es[:, 1] = torch.where(es[:, 0] == es[:, 1], (es[:, 1] + 1) % nA, es[:, 1])
    Gc = torch.empty((N, q), dtype=torch.float64, device=DEV).normal_(generator=gen).div_(math.sqrt(q))
    col, e = B // 2, N // 3
    a, b = (int(x) for x in es[e].cpu())
    # the winner's own column is positive at one endpoint and negative at the other
    U[:, a, col] = 0.2
    U[:, b, col] = -0.2
    win = np.zeros(6, np.int32)
    win[:3] = col, a, b
    win[4:6] = np.array([e], np.int64).view(np.int32)
    h = torch.empty((p, N), dtype=torch.float64, device=DEV)
    t = torch.empty((p, N), dtype=torch.float64, device=DEV)
    ea, eb = es[:, 0].long(), es[:, 1].long()
    for j in range(p):
        d = (XY[j, ea] - XY[j, eb]).double().square()
        h[j], t[j] = d[:, :q].sum(1), d[:, q:].sum(1)
    return dict(XY=XY, U=U, es=es, Gc=Gc, win=torch.as_tensor(win).to(DEV), h=h, t=t, col=col, a=a, b=b, e=e)


def _greedy_input(c, seed):
    gen = _gen(seed)
    E, w, deg = _graph_input(c, gen)
    cand = _candidates(c["n"], E, c["N"], gen)

    def normal(rows):
        out = torch.empty((rows, c["q"]), dtype=torch.float64, device=DEV)
        return out.normal_(generator=gen).div_(math.sqrt(c["q"]))

    Z, U, Gc = normal(c["n"]), normal(E.shape[0]), normal(c["N"])
    F = torch.zeros_like(Z).index_add_(0, E[:, 0], U).index_add_(0, E[:, 1], U, alpha=-1.0)
    return dict(E=E, deg=deg, cand=cand, sketch=(Z, F, Gc))


# ---- the cases ------------------------------------------------------------------------
def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "apply":
        gen = _gen(seed)
        E, w, _ = _graph_input(c, gen)
        dt = torch.float32 if c["prec"] == "mixed" else torch.float64
        x = torch.empty((c["n"], c["R"]), dtype=dt, device=DEV).normal_(generator=gen)
        return dict(kind=kind, op=pg.Op(_graph(c, E, w, 1e-2)), x=x[:, 0].contiguous() if c["R"] == 1 else x)
    if kind == "solve":
        i = _solve_input(c, seed)
        G = _graph(c, i["E"], i["w"], c["sigma"])
        op = pg.Op(G)
        for (a, b), we in zip(i["extra"].cpu().tolist(), i["wx"].cpu().tolist()):
            op.add(a, b, we)
        act, pos = prepare_active(i["active"], c["n"], G.device)
        return dict(kind=kind, op=op, W=i["W"], tau=torch.as_tensor(i["tau"], device=DEV), act=act, pos=pos,
                    tol=c["tol"], track=c["prec"] == "fp64", prec=c["prec"])
    if kind == "batch":
        ins = [(b, _solve_input(b, seed + 1000 * k)) for k, b in enumerate(_batch_cases(c))]
        return dict(kind=kind, ops=[pg.Op(_graph(b, i["E"], i["w"], b["sigma"])) for b, i in ins],
                    Ws=[i["W"] for _, i in ins], taus=[i["tau"] for _, i in ins],
                    acts=[i["active"].cpu().numpy() for _, i in ins], tol=c["tol"], prec=c["prec"])
    lib = _lib.load()
    if kind == "score":
        i = _score_input(c, seed)
        B, N = c["B"], c["N"]
        return dict(kind=kind, lib=lib, idx=torch.empty(B, dtype=torch.int64, device=DEV),
                    val=torch.empty(B, dtype=torch.float64, device=DEV),
                    every=torch.empty(N, dtype=torch.float64, device=DEV) if c["all"] else None,
                    tmp=torch.empty(lib.polar_topb_tmp_bytes(N, B), dtype=torch.uint8, device=DEV), p=c["p"], N=N, B=B,
                    obj=c["obj"], **i)
    if kind == "maintain":
        i = _maintain_input(c, seed)
        tmp = torch.empty(lib.polar_maintain_tmp_bytes(c["p"], c["rows"], c["q"]), dtype=torch.uint8, device=DEV)
        return dict(kind=kind, lib=lib, tmp=tmp, p=c["p"], nA=c["rows"], q=c["q"], N=c["N"], B=c["B"],
                    f32=1 if c["prec"] == "mixed" else 0, **i)
    i = _greedy_input(c, seed)
    return dict(kind=kind, G=_graph(c, i["E"], None, 1e-2), cand=i["cand"].cpu().numpy(), sketch=i["sketch"], c=c)


def run(state):
    kind = state["kind"]
    if kind == "apply":
        return state["op"](state["x"])
    if kind == "solve":
        X, h, _ = pg.msolve(state["op"], state["W"], state["tau"], state["act"], state["tol"], track=state["track"],
                            precision=state["prec"], active_pos=state["pos"])
        return [X, h] if state["track"] else [X]
    if kind == "batch":
        out = msolve_batch(state["ops"], state["Ws"], state["taus"], state["acts"], state["tol"],
                           precision=state["prec"])
        return [X for X, _, _ in out]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "score":
        s = state
        every = s["every"]
        _lib.check(s["lib"].polar_score_topb(s["h"].data_ptr(), s["t"].data_ptr(), s["tau"].data_ptr(),
                                             s["om"].data_ptr(), 1e-2, s["p"], s["N"], s["live"].data_ptr(), s["obj"],
                                             s["B"], s["idx"].data_ptr(), s["val"].data_ptr(),
                                             every.data_ptr() if every is not None else None, s["tmp"].data_ptr(),
                                             stream), "score_topb")
        return [s["idx"], s["val"]] + ([every] if every is not None else [])
    if kind == "maintain":
        s = state
        XY, q = s["XY"], s["q"]
        _lib.check(s["lib"].polar_maintain(XY.data_ptr(), 2 * q, XY[:, :, q:].data_ptr(), 2 * q, s["f32"], s["p"],
                                           s["nA"], q, s["U"].data_ptr(), s["f32"], s["B"], s["win"].data_ptr(),
                                           s["Gc"].data_ptr(), s["es"].data_ptr(), s["N"], s["h"].data_ptr(),
                                           s["t"].data_ptr(), s["tmp"].data_ptr(), stream), "maintain")
        return [XY, s["h"], s["t"]]
    c = state["c"]
    r = pg.polar(state["G"], state["cand"], c["k"], 0.5, q=c["q"], B=c["B"], tol=c["tol"], sketch=state["sketch"],
                 K=c["K"])
    return [np.array(r["sequence"]), np.array(r["marginals"])]


def _iterations(deg, n, sigma, tol):
    """A priori CG iteration count of the seed system: a quarter of the Chebyshev bound
    sqrt(kappa) / 2 ln(2 / tol), kappa from the structural cutoff of the degrees."""
    kappa = 2.0 * min(15000.0, math.sqrt(n * deg)) / sigma
    return 0.125 * math.sqrt(kappa) * math.log(2.0 / tol)


def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind == "batch":
        parts = [work(b) for b in _batch_cases(c)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    if kind in ("apply", "solve", "greedy"):
        n = c["n"]
        nnz = n * c["deg"]
        graph = 4.0 * (n + nnz) + (8.0 * nnz if c.get("weighted") else 0.0)
    if kind == "apply":
        es = 4 if c["prec"] == "mixed" else 8
        return {"bytes": graph + 2.0 * es * n * c["R"], "flops": 2.0 * (nnz + n) * c["R"]}
    if kind == "solve":
        es = 4 if c["prec"] == "mixed" else 8
        it = _iterations(c["deg"], n, c["sigma"], c["tol"])
        return {"bytes": graph + 8.0 * n * c["R"] + es * c["K"] * c["rows"] * c["R"],
                "flops": it * c["R"] * (2.0 * nnz + 10.0 * n + 1.5 * c["K"] * c["rows"])}
    if kind == "score":
        two = 2.0 if c["obj"] == 0 else 1.0
        return {"bytes": 8.0 * two * c["p"] * c["N"] + c["N"] + (8.0 * c["N"] if c["all"] else 0.0),
                "flops": 6.0 * c["p"] * c["N"]}
    if kind == "maintain":
        es = 4 if c["prec"] == "mixed" else 8
        return {"bytes": c["p"] * (4.0 * es * c["rows"] * c["q"] + es * c["rows"] + 32.0 * c["N"]) + 8.0 * c["N"],
                "flops": c["p"] * (8.0 * c["rows"] * c["q"] + 14.0 * c["N"])}
    it = _iterations(c["deg"], n, 1e-2, c["tol"])
    cols = 2 * c["q"] + c["k"] * c["B"]
    return {"bytes": graph + 16.0 * n * c["q"] + 8.0 * c["N"] * (c["q"] + 2), "flops": it * cols * (2.0 * nnz + 10.0 * n)}


# ---- 64-bit values in plain torch -------------------------------------------------------
def _csr(n, E, w, sigma, extra=None, wx=None):
    """L + sigma I (plus the added edges) as a torch FP64 CSR matrix."""
    w = torch.ones(E.shape[0], dtype=torch.float64, device=DEV) if w is None else w
    if extra is not None and extra.shape[0]:
        E, w = torch.cat([E, extra]), torch.cat([w, wx])
    i = torch.arange(n, device=DEV)
    rows = torch.cat([E[:, 0], E[:, 1], E[:, 0], E[:, 1], i])
    cols = torch.cat([E[:, 1], E[:, 0], E[:, 0], E[:, 1], i])
    vals = torch.cat([-w, -w, w, w, torch.full((n,), sigma, dtype=torch.float64, device=DEV)])
    return torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n, n)).coalesce().to_sparse_csr()


def _shifted_solves(M, W, tau, active, tol=1e-13):
    """(M + tau_j I)^-1 W on the active rows for every pole, and the squared norms of the whole
    columns: multi-shift CG in FP64 run far past the cases' tolerances."""
    tau = torch.as_tensor(tau, device=DEV)[:, None]
    theta = tau - tau[0]
    p, (n, R) = tau.shape[0], W.shape
    r, d = W.clone(), W.clone()
    rr = (r * r).sum(0)
    stop = tol * rr.sqrt()
    one = torch.ones((p, R), dtype=torch.float64, device=DEV)
    z, zp, P = one.clone(), one.clone(), r[active].expand(p, -1, -1).clone()
    X = torch.zeros_like(P)
    nh, ip, pn = torch.zeros_like(z), torch.zeros_like(z), rr.expand(p, -1).clone()
    a_old, b_old = torch.ones_like(rr), torch.zeros_like(rr)
    for it in range(20000):
        on = rr.sqrt() > stop
        if it % 16 == 0 and not bool(on.any()):
            break
        v = (M @ d).add_(d, alpha=float(tau[0]))
        a = torch.where(on, rr / (d * v).sum(0), 0.0)
        r -= a * v
        new = (r * r).sum(0)
        b = torch.where(on, new / rr, 0.0)
        # a pole of a column stands still once its own residual is far below the column's stop
        go = on & (z.abs() * rr.sqrt() > 1e-2 * stop)
        zn = torch.where(go, z / (1.0 + a * theta + a * b_old / a_old * (1.0 - z / zp)), z)
        f = zn / z
        aj, bj = torch.where(go, a * f, 0.0), torch.where(go, b * f * f, 1.0)
        nh += 2.0 * aj * ip + aj * aj * pn
        ip = bj * (ip + aj * pn)
        pn = torch.where(go, zn * zn * new + bj * bj * pn, pn)
        ra, zr = r[active], torch.where(go, zn, 0.0)
        for j in range(p):
            X[j].addcmul_(P[j], aj[j])
            P[j].mul_(bj[j]).addcmul_(ra, zr[j])
        zp, z = torch.where(go, z, zp), zn
        rr, a_old, b_old = torch.where(on, new, rr), torch.where(on, a, a_old), torch.where(on, b, b_old)
        d.mul_(b).add_(r)
    return X, nh


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "apply":
        return _exact_apply(c, seed)
    if kind == "solve":
        i = _solve_input(c, seed)
        M = _csr(c["n"], i["E"], i["w"], c["sigma"], i["extra"], i["wx"])
        X, h = _shifted_solves(M, i["W"], i["tau"], i["active"])
        return [X, h] if c["prec"] == "fp64" else [X]
    if kind == "batch":
        out = []
        for k, b in enumerate(_batch_cases(c)):
            i = _solve_input(b, seed + 1000 * k)
            out.append(_shifted_solves(_csr(b["n"], i["E"], i["w"], b["sigma"]), i["W"], i["tau"], i["active"])[0])
        return out
    if kind == "score":
        i = _score_input(c, seed)
        h, t, tau, om = i["h"], i["t"], i["tau"][:, None], i["om"][:, None]
        g = (om * h if c["obj"] == 2 else om * h / (1.0 + t + (1e-2 + tau) * h)).sum(0)
        top = torch.where(i["live"] != 0, g, torch.full_like(g, -math.inf))
        val, idx = torch.sort(top, descending=True, stable=True)
        return [idx[:c["B"]], val[:c["B"]]] + ([g] if c["all"] else [])
    if kind == "maintain":
        i = _maintain_input(c, seed)
        q, a, b = c["q"], i["a"], i["b"]
        XY, h, t = torch.empty(i["XY"].shape, dtype=torch.float64, device=DEV), i["h"], i["t"]
        ea, eb = i["es"][:, 0].long(), i["es"][:, 1].long()
        for j in range(c["p"]):
            X, Y, u = i["XY"][j, :, :q].double(), i["XY"][j, :, q:].double(), i["U"][j, :, i["col"]].double()
            xi, eta, D = X[a] - X[b], i["Gc"][i["e"]] - (Y[a] - Y[b]), 1.0 + u[a] - u[b]
            wx, wy, cc = X @ xi, Y @ eta, (u[ea] - u[eb]) / D
            h[j] = (h[j] - 2.0 * cc * (wx[ea] - wx[eb]) + cc * cc * (xi @ xi)).clamp_min(0.0)
            t[j] = (t[j] + 2.0 * cc * (wy[ea] - wy[eb]) + cc * cc * (eta @ eta)).clamp_min(0.0)
            XY[j, :, :q] = X - u[:, None] * (xi / D)
            XY[j, :, q:] = Y + u[:, None] * (eta / D)
        return [XY, h, t]
    i = _greedy_input(c, seed)
    Z, F, Gc = i["sketch"]
    sigma = 1e-2
    tau, om = _poles(0.5, c["K"], sigma, sigma + 2.0 * float(i["deg"].max()) + 4.0 * c["k"])
    M = _csr(c["n"], i["E"], None, sigma).to_dense()
    eye = torch.eye(c["n"], dtype=torch.float64, device=DEV)
    a, b = i["cand"][:, 0], i["cand"][:, 1]
    dead = torch.zeros(c["N"], dtype=torch.bool, device=DEV)
    seq, marg = [], []
    for _ in range(c["k"]):
        g = torch.zeros(c["N"], dtype=torch.float64, device=DEV)
        inv = [torch.linalg.inv(M + t * eye) for t in tau]
        for j, V in enumerate(inv):
            X, Y = V @ Z, V @ F
            h, t = (X[a] - X[b]).square().sum(1), (Y[a] - Y[b]).square().sum(1)
            g += om[j] * h / (1.0 + t + (sigma + tau[j]) * h)
        g[dead] = -math.inf
        short = torch.argsort(g, descending=True, stable=True)[:c["B"]]
        gq = torch.zeros(c["B"], dtype=torch.float64, device=DEV)
        for j, V in enumerate(inv):
            u = V[:, a[short]] - V[:, b[short]]
            k = torch.arange(c["B"], device=DEV)
            gq += om[j] * u.square().sum(0) / (1.0 + u[a[short], k] - u[b[short], k])
        best = int(torch.argmax(gq))
        e = int(short[best])
        seq.append(e)
        marg.append(float(gq[best]))
        dead[e] = True
        x, y = int(a[e]), int(b[e])
        M[x, x] += 1.0
        M[y, y] += 1.0
        M[x, y] -= 1.0
        M[y, x] -= 1.0
        F[x] += Gc[e]
        F[y] -= Gc[e]
    return [np.array(seq), np.array(marg)]


def _exact_apply(c, seed):
    """(L + sigma I) x of an apply case's inputs in FP64."""
    gen = _gen(seed)
    E, w, _ = _graph_input(c, gen)
    dt = torch.float32 if c["prec"] == "mixed" else torch.float64
    x = torch.empty((c["n"], c["R"]), dtype=dt, device=DEV).normal_(generator=gen).double()
    y = _csr(c["n"], E, w, 1e-2) @ x
    return y[:, 0].contiguous() if c["R"] == 1 else y
