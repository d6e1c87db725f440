"""Whole solves in one launch (thread-block clusters): row classes, widths, pole counts and
active sets at their edges, against a dense FP64 solve."""
import numpy as np
import pytest

from polar_b200.synth import chung_lu

pytestmark = pytest.mark.gpu

# ||r|| <= tol ||w|| with eigenvalues from 2e-2: FP64 at 1e-12 is far below 1e-9; mixed
# iterates are FP32 at 1e-7
BOUND = {"fp64": (1e-12, 1e-9), "mixed": (1e-7, 1e-4)}


def _star(n, arms):
    """Vertices 0, 1, 2, ... with arms[i] leaves each (rows of one lane, 8 lanes, a warp, a CTA),
    the leaves chained, the last vertices isolated."""
    out, at = [], len(arms)
    for i, a in enumerate(arms):
        out += [(i, at + k) for k in range(a)]
        at += a
    out += [(i, i + 1) for i in range(len(arms), at - 1)]
    assert at <= n
    return np.array(out)


GRAPHS = {
    "tiny": lambda: (3, np.array([[0, 1], [1, 2]])),
    "row33": lambda: (33, chung_lu(33, 3.0, 2.5, 0, min_degree=1)),
    "plain": lambda: (2000, chung_lu(2000, 6.0, 2.5, 0, min_degree=1)),
    "star": lambda: (3500, _star(3500, [17, 16, 256, 257, 1024, 1025])),
    "none": lambda: (40, np.zeros((0, 2), np.int64)),
}


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("graph,R,p,weighted,active", [
    ("tiny", 1, 1, False, 1), ("row33", 3, 17, False, 33), ("row33", 64, 2, True, 5), ("plain", 1, 16, False, 2),
    ("plain", 64, 40, False, 2000), ("plain", 17, 16, True, 700), ("star", 5, 3, False, 3500), ("star", 2, 33, True, 100),
    ("none", 4, 2, False, 40)])
def test_against_dense(prec, graph, R, p, weighted, active):
    import torch
    import polar_b200 as pg
    from polar_b200 import _lib
    tol, bound = BOUND[prec]
    n, E = GRAPHS[graph]()
    rng = np.random.default_rng(R + p)
    w = rng.uniform(0.3, 2.0, len(E)) if weighted else None
    G = pg.Graph(n, E, 2e-2, weights=w)
    op = pg.Op(G)
    M = np.asarray(G.M0.get().todense())
    op.add(0, n - 1, 0.7)  # an added edge
    for a, b, v in ((0, 0, 0.7), (n - 1, n - 1, 0.7), (0, n - 1, -0.7), (n - 1, 0, -0.7)):
        M[a, b] += v
    W = rng.normal(size=(n, R))
    if R > 2:
        W[:, 1] = 0.0  # a column that is solved from the start
    tau = np.concatenate([[0.0], np.geomspace(1e-2, 1e3, p - 1)]) if p > 1 else np.zeros(1)
    act = np.sort(rng.permutation(n)[:active])
    lib = _lib.load()
    before = lib.polar_launch_count()
    X, h, it = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    assert lib.polar_launch_count() - before == 3  # row order, lists, the solve
    X2, h2, it2 = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    assert torch.equal(X, X2) and torch.equal(h, h2) and np.array_equal(it, it2)
    Md, Wd = torch.as_tensor(M, device="cuda"), torch.as_tensor(W, device="cuda")
    rows = torch.as_tensor(act, device="cuda")
    for j, t in enumerate(tau):
        full = torch.linalg.solve(Md + t * torch.eye(n, dtype=torch.float64, device="cuda"), Wd)
        ref = torch.linalg.norm(full)
        assert float(torch.linalg.norm(X[j].double() - full[rows]) / ref) < bound
        hw = full.square().sum(0)
        assert float(((h[j] - hw).abs() / hw.clamp_min(1e-300)).max()) < bound
    if R > 2:
        assert it[1] == 0


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_iteration_cap_and_nonfinite(prec):
    import torch
    import polar_b200 as pg
    from polar_b200 import _lib
    n, E = GRAPHS["plain"]()
    op = pg.Op(pg.Graph(n, E, 1e-2))
    rng = np.random.default_rng(0)
    W = rng.normal(size=(n, 5))
    tau = np.array([0.0, 1.0])
    for maxit in (0, 1, 15, 16, 17):
        out = torch.full((2, 3, 5), 7.0, dtype=torch.float64, device="cuda")
        with pytest.raises(_lib.PolarError, match="iteration cap"):
            pg.msolve(op, W, tau, [0, 5, 9], 1e-12, maxit=maxit, precision=prec, out=out)
        assert bool((out != 7.0).all())  # the iterates reached so far
    W[3, 2] = np.nan
    with pytest.raises(_lib.PolarError) as e:
        pg.msolve(op, W, tau, [0, 5, 9], 1e-8, precision=prec)
    assert e.value.status == _lib.POLAR_ERR_NONFINITE
