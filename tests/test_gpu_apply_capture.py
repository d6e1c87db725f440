"""Operator applies under stream capture after an eager call of another width."""
import numpy as np
import pytest

from polar_b200.synth import chung_lu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [3000, 250_000])
@pytest.mark.parametrize("layout,eager,captured", [
    (kind, e, c) for kind in ("weighted", "rows") for e, c in ((16, 14), (16, 1), (14, 16), (1, 16), (1, 14), (14, 3))
] + [("sliced", e, c) for e, c in ((16, 14), (14, 16), (16, 9), (13, 16), (4, 3), (3, 4), (2, 1), (20, 32))])
def test_apply(prec, n, layout, eager, captured):
    """Weighted graphs, and others with the sliced-ELL layout off ("rows"), need nothing new for
    another width, so one eager call prepares them all; a sliced-ELL layout is one per power of
    two of columns."""
    import torch
    import polar_b200 as pg
    from polar_b200 import _lib
    E = chung_lu(n, 9.0, 2.1, 3, min_degree=1)  # rows above and below every partition's threshold
    w = np.random.default_rng(1).uniform(0.5, 1.5, len(E)) if layout == "weighted" else None
    G = pg.Graph(n, E, 5e-1, weights=w)
    op = pg.Op(G)
    if layout == "rows":
        _lib.load().polar_set_sell(0)
    try:
        _check(torch, G, op, prec, n, eager, captured)
    finally:
        _lib.load().polar_set_sell(1)


def _check(torch, G, op, prec, n, eager, captured):
    dt = torch.float64 if prec == "fp64" else torch.float32
    gen = torch.Generator("cuda").manual_seed(n)
    op(torch.randn((n, eager), dtype=dt, device="cuda", generator=gen))
    x = torch.randn((n, captured), dtype=dt, device="cuda", generator=gen)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = op(x)
    eager_first = op(x)  # before any replay: nothing of it was left to the graph
    M = G.M0.get().tocsr()
    A = torch.sparse_csr_tensor(torch.as_tensor(M.indptr), torch.as_tensor(M.indices), torch.as_tensor(M.data),
                                size=M.shape, dtype=torch.float64).cuda()
    size = torch.sparse_csr_tensor(A.crow_indices(), A.col_indices(), A.values().abs(), size=M.shape)
    # a row of d terms summed in the row's precision: d roundings of at most |A| |x|
    bound = (int(np.diff(M.indptr).max()) + 4) * (2.0 ** -52 if prec == "fp64" else 2.0 ** -23)
    for _ in range(2):
        x.copy_(torch.randn((n, captured), dtype=dt, device="cuda", generator=gen))
        g.replay()
        torch.cuda.synchronize()
        assert float(((y.double() - A @ x.double()).abs() / (size @ x.double().abs())).max()) < bound
    assert torch.isfinite(eager_first).all()
