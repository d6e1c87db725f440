"""256-bit row accesses of the solver and of the operator apply: block widths around the lane
rule, weighted and plain graphs, workspaces and blocks that start at any 16 bytes."""
import numpy as np
import pytest

from polar_b200.synth import chung_lu

pytestmark = pytest.mark.gpu

N = 61000  # above the cluster solver's row limit


def _graph(weighted):
    import polar_b200 as pg
    E = chung_lu(N, 5.0, 2.3, 3, min_degree=1)
    w = np.random.default_rng(1).uniform(0.5, 1.5, len(E)) if weighted else None
    return pg.Graph(N, E, 5e-1, weights=w)


def _csr(G):
    import torch
    M = G.M0.get().tocsr()
    return torch.sparse_csr_tensor(torch.as_tensor(M.indptr), torch.as_tensor(M.indices), torch.as_tensor(M.data),
                                   size=M.shape, dtype=torch.float64).cuda()


# ||W - M x|| <= tol ||W|| for the recurred residual; the true one differs from it by rounding:
# far below tol in FP64 (1e-8), by FP32 products and iterates in mixed (6e-8 of |M| |x| per
# product: |M| / sigma ~ 3e3 bounds it by 2e-4)
@pytest.mark.parametrize("prec,tol,bound", [("fp64", 1e-8, 1.5e-8), ("mixed", 1e-6, 2e-4)])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("R", [1, 2, 4, 8, 15, 16, 33, 64, 65, 128])
def test_solve_residual_and_workspace_offset(prec, tol, bound, weighted, R, monkeypatch):
    import torch
    import polar_b200 as pg
    from polar_b200 import solver
    G = _graph(weighted)
    op = pg.Op(G)
    W = torch.randn((N, R), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(R))
    tau = np.array([0.0, 2.0])
    act = np.arange(N)
    X, _, it = pg.msolve(op, W, tau, act, tol, precision=prec)
    A = _csr(G)
    for j, t in enumerate(tau):
        x = X[j].double()
        r = W - (A @ x + t * x)
        assert float((r.norm(dim=0) / W.norm(dim=0)).max()) < bound
    # a workspace that starts 16 bytes off the alignment of the rows
    monkeypatch.setattr(solver, "workspace",
                        lambda nb, dev: torch.empty(int(nb) + 16, dtype=torch.uint8, device=dev)[16:])
    X2, _, it2 = pg.msolve(op, W, tau, act, tol, precision=prec)
    assert torch.equal(X, X2) and np.array_equal(it, it2)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("R", [8, 16, 32, 64, 128])
def test_apply_at_any_16_bytes(prec, R):
    import torch
    import polar_b200 as pg
    if prec == "fp64" and R > 64:
        pytest.skip("64 columns at most in FP64")
    G = _graph(False)
    op = pg.Op(G)
    op.add(3, N - 1, 0.7)
    dt = torch.float64 if prec == "fp64" else torch.float32
    off = 16 // torch.empty((), dtype=dt).element_size()
    buf = torch.randn(N * R + off, dtype=dt, device="cuda", generator=torch.Generator("cuda").manual_seed(7))
    x = buf[off:].view(N, R)
    assert x.data_ptr() % 32 == 16
    want = _csr(G) @ x.double()
    d = 0.7 * (x[3].double() - x[N - 1].double())
    want[3] += d
    want[N - 1] -= d
    scale = want.abs().max()
    # one rounding of a row sum per entry: 2^-53 or 2^-24 of the largest row, a few terms over
    bound = 1e-14 if prec == "fp64" else 2e-7
    for v in (x, x.clone()):
        assert float((op(v).double() - want).abs().max() / scale) < bound


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("own", [256, 8])  # the graph's own partition: coarser and finer than the rule's
@pytest.mark.parametrize("R", [1, 2, 3, 4, 12, 14, 16, 20, 28, 31, 60])
def test_apply_partitions(prec, weighted, own, R):
    import torch
    import polar_b200 as pg
    n = 5000
    E = chung_lu(n, 9.0, 2.1, 3, min_degree=1)  # rows of up to a few hundred neighbours
    w = np.random.default_rng(1).uniform(0.5, 1.5, len(E)) if weighted else None
    G = pg.Graph(n, E, 5e-1, weights=w, heavy_thresh=own)
    op = pg.Op(G)
    op.add(3, n - 1, 0.7)
    dt = torch.float64 if prec == "fp64" else torch.float32
    A = _csr(G).to_dense()
    for a, b, v in ((3, 3, 0.7), (n - 1, n - 1, 0.7), (3, n - 1, -0.7), (n - 1, 3, -0.7)):
        A[a, b] += v
    # a row of d <= 500 terms summed in the row's precision: d roundings of at most |A| |x|
    bound = 500 * (2.0 ** -52 if prec == "fp64" else 2.0 ** -23)
    for width in (R, 3, R):  # another partition and its scratch between two calls
        x = torch.randn((n, width), dtype=dt, device="cuda", generator=torch.Generator("cuda").manual_seed(width))
        want = A @ x.double()
        size = A.abs() @ x.double().abs()
        assert float(((op(x).double() - want).abs() / size).max()) < bound


# long lists of added edges on the kernel-per-phase driver; bounds as above
@pytest.mark.parametrize("prec,tol,bound", [("fp64", 1e-8, 1.5e-8), ("mixed", 1e-6, 2e-4)])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("R,m", [(1, 600), (5, 40), (16, 700), (64, 5), (64, 900)])
def test_added_edges_residual(prec, tol, bound, weighted, R, m):
    import torch
    import polar_b200 as pg
    G = _graph(weighted)
    op = pg.Op(G)
    rng = np.random.default_rng(m)
    pairs = rng.permutation(N)[:2 * m].reshape(m, 2)
    hub = int(np.argmax(np.diff(G._indptr_h)))
    pairs = np.vstack([pairs, [[hub, k] for k in (7, 11, 13) if k != hub]])  # several at a heavy row
    w = rng.uniform(0.2, 2.0, len(pairs))
    for (a, b), we in zip(pairs, w):
        op.add(int(a), int(b), float(we))
    gen = torch.Generator("cuda").manual_seed(R)
    W = torch.randn((N, R), dtype=torch.float64, device="cuda", generator=gen)
    tau = np.array([0.0, 2.0])
    X, _, _ = pg.msolve(op, W, tau, np.arange(N), tol, precision=prec)
    A = _csr(G)
    a, b = (torch.as_tensor(pairs[:, k], device="cuda") for k in (0, 1))
    wd = torch.as_tensor(w, device="cuda")[:, None]
    for j, t in enumerate(tau):
        x = X[j].double()
        r = W - (A @ x + t * x)
        d = wd * (x[a] - x[b])
        r.index_add_(0, a, d, alpha=-1.0).index_add_(0, b, d)
        assert float((r.norm(dim=0) / W.norm(dim=0)).max()) < bound
