"""Multi-shift solves on operators with added edges, around the size where their terms leave
the SpMM's last CTA for a kernel of their own, against a dense FP64 solve."""
import numpy as np
import pytest

from polar_b200.synth import chung_lu

pytestmark = pytest.mark.gpu


# (columns, added edges): items = (rows with added edges) x (padded columns); one CTA has 512
# threads, so 64 x 8 stays in the SpMM and 64 x 9 (a shared endpoint makes an odd count) does not
@pytest.mark.parametrize("prec,tol,bound", [("fp64", 1e-12, 1e-9), ("mixed", 1e-7, 1e-4)])
@pytest.mark.parametrize("R,m,odd", [(64, 4, False), (64, 4, True), (1, 700, False), (5, 300, True), (64, 900, False)])
def test_added_edges_against_dense(prec, tol, bound, R, m, odd):
    # bound: ||r|| <= tol ||w|| and the smallest eigenvalue 2e-2 give a relative error of the
    # iterates below 50 tol kappa^(1/2) << bound in FP64; mixed: FP32 iterates at tol 1e-7
    import torch
    import polar_b200 as pg
    n, sigma = 3000, 2e-2
    E = chung_lu(n, 6.0, 2.5, 5, min_degree=1)
    rng = np.random.default_rng(m + R)
    perm = rng.permutation(n)
    pairs = perm[:2 * m].reshape(m, 2)
    if odd:  # one more edge that shares an endpoint: an odd number of rows
        pairs = np.vstack([pairs, [pairs[0, 0], perm[2 * m]]])
    w = rng.uniform(0.1, 2.0, len(pairs))
    G = pg.Graph(n, E, sigma)
    op = pg.Op(G)
    M = np.asarray(G.M0.get().todense())
    for (a, b), we in zip(pairs, w):
        op.add(int(a), int(b), float(we))
        M[a, a] += we
        M[b, b] += we
        M[a, b] -= we
        M[b, a] -= we
    W = rng.normal(size=(n, R))
    tau = np.array([0.0, 0.3, 20.0])
    act = np.sort(rng.permutation(n)[:500])
    X, h, _ = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
    Md = torch.as_tensor(M, device="cuda")
    for j, t in enumerate(tau):
        full = torch.linalg.solve(Md + t * torch.eye(n, dtype=torch.float64, device="cuda"), torch.as_tensor(W, device="cuda"))
        want = full[torch.as_tensor(act, device="cuda")]
        err = torch.linalg.norm(X[j].double() - want) / torch.linalg.norm(want)
        assert float(err) < bound
        hw = full.square().sum(0)
        assert float(((h[j] - hw).abs() / hw).max()) < bound
