"""Solver workspaces hold the cluster solver's regions where it runs, and nowhere else."""
import contextlib

import numpy as np
import pytest

from polar_b200.synth import chung_lu

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _residual(lib, bits):
    lib.polar_set_mixed_residual(bits)
    try:
        yield
    finally:
        lib.polar_set_mixed_residual(64)


def _record(_lib, n, nnz, weighted=False):
    g = _lib.PolarGraph()  # the query reads sizes and whether there are weights
    g.n, g.nnz = n, nnz
    if weighted:
        g.d_wts = g.d_diag = 256
    return g


def _phases(solver, ask):
    was = solver.set_cluster_solver(False)
    try:
        return ask()
    finally:
        solver.set_cluster_solver(was)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("weighted", [False, True])
def test_sizes(prec, weighted):
    from polar_b200 import _lib, solver
    lib = _lib.load()
    pc = solver.precision_code(prec)
    ts = 4 if prec == "mixed" else 8
    n, R, p, nA = 20000, 64, 24, 15000
    g = _record(_lib, n, 130_000, weighted)
    # rows r, d, v (and the direction's remainder), 16 history slots, P and X; 16 MiB for the rest
    vec = n * R * (8 + 2 * ts + (4 if ts == 4 else 0)) + (16 + 2 * p) * nA * R * ts
    batch = lib.polar_msolve_batch_workspace_bytes(g, pc, R, p, nA)
    assert vec < batch < vec + (16 << 20)
    ask = lambda gg=g, pp=p, aa=nA: lib.polar_msolve_workspace_bytes(gg, pc, R, pp, aa)
    assert vec < _phases(solver, ask) < vec + (16 << 20)
    if prec == "mixed":
        with _residual(lib, 32):
            assert vec < ask() < vec + (16 << 20)
    # a shape that the cluster solver does not take: no lists of its 2e7 neighbours
    dense = _record(_lib, 50000, 20_000_000, weighted)
    assert ask(dense) == _phases(solver, lambda: ask(dense))
    # one that it takes: FP64 iterates and the lists
    small = _record(_lib, 2000, 12_000, weighted)
    more = ask(small, 8, 1000) - _phases(solver, lambda: ask(small, 8, 1000))
    assert more >= 8 * 1000 * R * (8 - ts) + 3 * 12_000 * 2


@pytest.mark.parametrize("prec,tol,bound", [("fp64", 1e-12, 1e-9), ("mixed", 1e-7, 1e-4)])
def test_workspace_of_other_settings(prec, tol, bound, monkeypatch):
    """A workspace sized for the kernels per phase stays enough when the setting has changed."""
    import torch
    import polar_b200 as pg
    from polar_b200 import _lib, solver
    lib = _lib.load()
    n, R = 2000, 16
    op = pg.Op(pg.Graph(n, chung_lu(n, 6.0, 2.5, 0, min_degree=1), 2e-2))
    W = np.random.default_rng(0).normal(size=(n, R))
    tau, act = np.array([0.0, 1.0]), np.arange(0, n, 3)
    was = solver.set_cluster_solver(False)
    need = []
    monkeypatch.setattr(solver, "workspace", lambda nb, dev: need.append(int(nb)) or torch.empty(int(nb), dtype=torch.uint8, device=dev))
    try:
        X, _, _ = pg.msolve(op, W, tau, act, tol, precision=prec)
    finally:
        solver.set_cluster_solver(was)
    monkeypatch.setattr(solver, "workspace", lambda nb, dev: need.append(int(nb)) or torch.empty(need[0], dtype=torch.uint8, device=dev))
    X2, _, _ = pg.msolve(op, W, tau, act, tol, precision=prec)
    assert need[1] > need[0] and torch.equal(X, X2)
    monkeypatch.setattr(solver, "workspace", lambda nb, dev: torch.empty(need[0] - 1, dtype=torch.uint8, device=dev))
    with pytest.raises(_lib.PolarError) as e:
        pg.msolve(op, W, tau, act, tol, precision=prec)
    assert e.value.status == _lib.POLAR_ERR_WORKSPACE


# shapes far from the line between the drivers: (n, nnz, rows with added edges, R, poles, active)
@pytest.mark.parametrize("prec,shape,taken", [
    ("fp64", (2000, 12000, 0, 1, 16, 2), True), ("fp64", (2000, 11000, 2000, 64, 16, 1000), True),
    ("fp64", (20000, 110000, 6500, 16, 16, 1000), True), ("mixed", (20000, 110000, 6500, 128, 16, 1000), True),
    ("fp64", (27647, 450000, 3929, 64, 15, 569), False), ("mixed", (50351, 463000, 2965, 48, 22, 3), False),
    ("mixed", (50000, 274000, 7900, 64, 16, 1000), False), ("mixed", (50000, 1500000, 0, 64, 16, 1000), False),
    ("fp64", (317000, 2000000, 0, 1, 16, 2), False)])
def test_choice_between_drivers(prec, shape, taken):
    from polar_b200 import _lib, solver
    lib = _lib.load()
    n, nnz, nx, R, p, nA = shape
    g = _record(_lib, n, nnz)
    g.nx = nx
    ask = lambda: lib.polar_msolve_workspace_bytes(g, solver.precision_code(prec), R, p, nA)
    assert (ask() > _phases(solver, ask)) == taken
