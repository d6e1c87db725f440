"""Cluster solves of graphs with many wide rows, on warps and on whole CTAs, against a dense FP64
solve."""
import numpy as np
import pytest

from polar_b200.synth import chung_lu

pytestmark = pytest.mark.gpu

# ||r|| <= tol ||w|| with eigenvalues from 1e-1: FP64 at 1e-12 is far below 1e-9; mixed
# iterates are FP32 at 1e-7
BOUND = {"fp64": (1e-12, 1e-9), "mixed": (1e-7, 1e-4)}


def _hubs(n, degrees):
    """A sparse graph with len(degrees) vertices of at least so many neighbours."""
    rng = np.random.default_rng(n)
    h = len(degrees)
    X = [np.stack([np.full(d, i), rng.choice(np.arange(h, n), d, replace=False)], 1) for i, d in enumerate(degrees)]
    return np.unique(np.sort(np.vstack([chung_lu(n, 5.0, 2.5, 1, min_degree=1)] + X), 1), axis=0)


def _dense(n, d):
    E = np.stack(np.triu_indices(n, 1), 1)
    return E[np.random.default_rng(n).random(len(E)) < d / (n - 1)]


GRAPHS = {
    "many": lambda: (2500, _dense(2500, 1100)),                       # every row above a warp's 8 lanes
    "one each": lambda: (12000, _hubs(12000, [9000] * 7 + [3000] * 9)),    # a CTA's widest row, the next on warps
    "two each": lambda: (12000, _hubs(12000, [9500] * 3 + [4200, 1025, 1024])),
    "widths": lambda: (9000, _hubs(9000, [8500, 4097, 4096, 4095, 2049, 2048, 2047, 257, 256])),
}


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("graph,R", [("many", 1), ("one each", 1), ("one each", 16), ("two each", 64), ("two each", 5), ("widths", 2)])
def test_against_dense(prec, weighted, graph, R):
    import torch
    import polar_b200 as pg
    from polar_b200 import solver
    tol, bound = BOUND[prec]
    n, E = GRAPHS[graph]()
    rng = np.random.default_rng(R)
    G = pg.Graph(n, E, 1e-1, weights=rng.uniform(0.3, 2.0, len(E)) if weighted else None)
    op = pg.Op(G)
    W = rng.normal(size=(n, R))
    tau = np.array([0.0, 10.0])
    act = np.sort(rng.permutation(n)[:n // 2])
    X, h, it = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    X2, h2, it2 = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    assert torch.equal(X, X2) and torch.equal(h, h2) and np.array_equal(it, it2)
    M, Wd = torch.as_tensor(G.M0.get().todense(), device="cuda"), torch.as_tensor(W, device="cuda")
    rows = torch.as_tensor(act, device="cuda")
    for j, t in enumerate(tau):
        full = torch.cholesky_solve(Wd, torch.linalg.cholesky(M + t * torch.eye(n, dtype=torch.float64, device="cuda")))
        assert float(torch.linalg.norm(X[j].double() - full[rows]) / torch.linalg.norm(full)) < bound
        hw = full.square().sum(0)
        assert float(((h[j] - hw).abs() / hw).max()) < bound
    # the kernels per phase agree
    was = solver.set_cluster_solver(False)
    try:
        Xp, _, _ = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    finally:
        solver.set_cluster_solver(was)
    assert float((Xp - X).double().norm() / X.double().norm()) < bound
