"""The kernel-per-phase driver on small graphs, which the cluster solver otherwise takes: heavy
rows, added edges on both sides of the size where they leave the SpMM's last CTA, iteration caps
and bad input, against a dense FP64 solve."""
import contextlib

import numpy as np
import pytest

from polar_b200.synth import chung_lu

pytestmark = pytest.mark.gpu

# ||r|| <= tol ||w|| with eigenvalues from 2e-2: FP64 at 1e-12 is far below 1e-9; mixed
# iterates are FP32 at 1e-7
BOUND = {"fp64": (1e-12, 1e-9), "mixed": (1e-7, 1e-4)}


@contextlib.contextmanager
def _phases():
    """Kernels per phase inside; yields a dict that holds the launches per class afterwards."""
    from polar_b200 import _lib, solver
    lib = _lib.load()
    was = solver.set_cluster_solver(False)
    lib.polar_set_kernel_timing(1)
    seen = {}
    try:
        yield seen
        seen.update({k: v[0] for k, v in _lib.kernel_timing().items()})
    finally:
        lib.polar_set_kernel_timing(0)
        solver.set_cluster_solver(was)


def _check(pg, n, E, w, added, R, prec, seen_for):
    import torch
    tol, bound = BOUND[prec]
    rng = np.random.default_rng(R + len(added))
    G = pg.Graph(n, E, 2e-2, weights=w)
    op = pg.Op(G)
    M = np.asarray(G.M0.get().todense())
    for a, b, we in added:
        op.add(int(a), int(b), float(we))
        for i, j, v in ((a, a, we), (b, b, we), (a, b, -we), (b, a, -we)):
            M[i, j] += v
    W = rng.normal(size=(n, R))
    tau = np.array([0.0, 0.3, 20.0])
    act = np.sort(rng.permutation(n)[:n // 3])
    with _phases() as seen:
        X, h, it = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
        X2, h2, it2 = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    assert torch.equal(X, X2) and torch.equal(h, h2) and np.array_equal(it, it2)
    assert seen["cluster"] == 0 and min(seen[k] for k in ("spmm", "resid", "dir", "flush")) > 0
    seen_for(seen)
    Md, Wd = torch.as_tensor(M, device="cuda"), torch.as_tensor(W, device="cuda")
    rows = torch.as_tensor(act, device="cuda")
    for j, t in enumerate(tau):
        full = torch.linalg.solve(Md + t * torch.eye(n, dtype=torch.float64, device="cuda"), Wd)
        assert float(torch.linalg.norm(X[j].double() - full[rows]) / torch.linalg.norm(full)) < bound
        hw = full.square().sum(0)
        assert float(((h[j] - hw).abs() / hw).max()) < bound
    # the cluster solver takes the same call again
    lib = pg._lib.load()
    before = lib.polar_launch_count()
    Xc, _, _ = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    assert lib.polar_launch_count() - before == 3
    assert float(torch.linalg.norm((Xc - X).double()) / torch.linalg.norm(X.double())) < bound


# one CTA's 512 threads take an item = (row with added edges, padded column) each: 8 rows of 64
# columns stay in the SpMM, 9 do not
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("R,m,odd,split", [(64, 4, False, False), (64, 4, True, True), (64, 1, False, False),
                                           (5, 32, False, False), (5, 32, True, True), (64, 300, False, True)])
def test_added_edges(prec, R, m, odd, split):
    import polar_b200 as pg
    n = 3000
    E = chung_lu(n, 6.0, 2.5, 5, min_degree=1)
    rng = np.random.default_rng(m)
    perm = rng.permutation(n)
    pairs = perm[:2 * m].reshape(m, 2)
    if odd:  # one more row, with a shared endpoint
        pairs = np.vstack([pairs, [pairs[0, 0], perm[2 * m]]])
    added = [(a, b, w) for (a, b), w in zip(pairs, rng.uniform(0.1, 2.0, len(pairs)))]
    _check(pg, n, E, None, added, R, prec, lambda s: (s["added"] > 0) == split or pytest.fail(str(s)))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("R", [1, 3, 16, 33, 64])
def test_heavy_rows(prec, weighted, R):
    import polar_b200 as pg
    n = 2500
    E = chung_lu(n, 8.0, 2.1, 3, min_degree=1)
    hubs = [(i, 100 * i + k) for i, d in ((0, 31), (1, 32), (2, 33), (3, 64), (4, 65), (5, 700)) for k in range(900, 900 + d)]
    E = np.unique(np.sort(np.vstack([E, hubs]), 1), axis=0)
    w = np.random.default_rng(0).uniform(0.3, 2.0, len(E)) if weighted else None
    _check(pg, n, E, w, [(0, n - 1, 0.7)], R, prec, lambda s: None)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_iteration_cap_and_nonfinite(prec):
    import torch
    import polar_b200 as pg
    from polar_b200 import _lib
    n = 2000
    op = pg.Op(pg.Graph(n, chung_lu(n, 6.0, 2.5, 0, min_degree=1), 1e-2))
    W = np.random.default_rng(0).normal(size=(n, 5))
    tau = np.array([0.0, 1.0])
    with _phases() as seen:
        for maxit in (1, 15, 16, 17, 40):
            out = torch.full((2, 3, 5), 7.0, dtype=torch.float64, device="cuda")
            with pytest.raises(_lib.PolarError, match="iteration cap"):
                pg.msolve(op, W, tau, [0, 5, 9], 1e-12, maxit=maxit, precision=prec, out=out)
            assert bool((out != 7.0).all())  # the iterates reached so far
        W[3, 2] = np.nan
        with pytest.raises(_lib.PolarError) as e:
            pg.msolve(op, W, tau, [0, 5, 9], 1e-8, precision=prec)
        assert e.value.status == _lib.POLAR_ERR_NONFINITE
    assert seen["cluster"] == 0 and seen["resid"] > 0


def test_setting_belongs_to_the_thread():
    import threading
    from polar_b200 import solver
    got = []
    assert solver.set_cluster_solver(False) is True
    try:
        t = threading.Thread(target=lambda: got.append(solver.set_cluster_solver(True)))
        t.start()
        t.join()
        assert got == [True]
    finally:
        assert solver.set_cluster_solver(True) is False


@pytest.mark.parametrize("prec,R", [("fp64", 16), ("mixed", 64)])
def test_tuner_times_the_kernels_per_phase(prec, R):
    import polar_b200 as pg
    from polar_b200 import _lib, autotune, solver
    lib = _lib.load()
    op = pg.Op(pg.Graph(4000, chung_lu(4000, 8.0, 2.1, 21, min_degree=1), 1e-2))
    lib.polar_set_kernel_timing(1)
    try:
        res = autotune.tune_msolve(op, R, prec, iters=16, reps=1, heavy_mult=(4, 32))
        seen = {k: v[0] for k, v in _lib.kernel_timing().items()}
    finally:
        lib.polar_set_kernel_timing(0)
    # two runs of 16 iterations per layout
    assert seen["cluster"] == 0 and seen["resid"] == 32 * len(res["table"])
    assert solver.set_cluster_solver(True) is True


@pytest.mark.parametrize("prec,R", [("fp64", 1), ("fp64", 16), ("mixed", 16), ("mixed", 64)])
def test_recorded_layouts_give_the_same_solve(prec, R):
    """Lane bytes, sliced-ELL or CSR rows and the heavy-row threshold change the order of sums only."""
    import polar_b200 as pg
    from polar_b200 import autotune
    n = 4000
    E = chung_lu(n, 8.0, 2.1, 21, min_degree=1)
    G = pg.Graph(n, E, 2e-2)
    op = pg.Op(G)
    assert np.diff(G._indptr_h).max() > 100  # chunked at two of the thresholds
    rng = np.random.default_rng(5)
    W, tau, act = rng.normal(size=(n, R)), np.array([0.0, 0.3, 20.0]), np.sort(rng.permutation(n)[:700])
    tol, bound = BOUND[prec]
    with _phases() as seen:
        X, h, _ = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
        for lanes in (16, 32, 64):
            for sell in (0, 1):
                for thresh in (16, 100, 5000):
                    autotune.record(G, prec, R, (lanes, sell, thresh))
                    X2, h2, _ = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
                    assert float((X2 - X).double().norm() / X.double().norm()) < bound, (lanes, sell, thresh)
                    assert float(((h2 - h).abs() / h).max()) < bound, (lanes, sell, thresh)
    assert seen["cluster"] == 0 and seen["spmm"] > 0
