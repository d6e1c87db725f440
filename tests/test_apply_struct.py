"""The graph record of an operator apply: what it builds on the host, and when."""
import numpy as np
import pytest

from polar_b200.synth import chung_lu


def _edges(n):
    rng = np.random.default_rng(0)
    hub = np.stack([np.zeros(600, np.int64), rng.permutation(n - 1)[:600] + 1], 1)
    return np.vstack([hub, [[1, 2], [2, 3]]]) if n > 100_000 else chung_lu(n, 9.0, 2.1, 3, min_degree=1)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,own", [(3000, 256), (3000, 8), (1_000_001, 256), (1_000_001, 8)])
def test_no_row_blocks_in_an_apply(monkeypatch, weighted, n, own):
    """Neither the sliced-ELL nor the row-loop kernel reads row blocks, so no apply of any width
    builds them; the panel kernel's (weighted graphs) come with the graph."""
    import polar_b200 as pg
    from polar_b200 import _lib, graph
    lib = _lib.load()
    E = _edges(n)
    w = np.linspace(0.5, 2.0, len(E)) if weighted else None
    op = pg.Op(pg.Graph(n, E, 1e-2, weights=w, heavy_thresh=own, device="cpu"))
    monkeypatch.setattr(graph, "row_blocks", lambda *a, **k: pytest.fail("row blocks built in an apply"))
    deg = np.diff(op.G._indptr_h)
    for prec, vec in ((_lib.POLAR_FP64, 2), (_lib.POLAR_MIXED, 4)):
        for R in ((1, 3, 8, 14, 16, 20) if n < 10_000 else (1, 16)):
            g = op._struct_for(lib, prec, R)
            panel = weighted and R % vec == 0 and R & (R - 1) == 0
            assert (g.nrb > 0) == panel
            # every row is in one place: a chunked one, or a light one of the layout that is read
            assert g.nheavy == (deg > g.heavy_thresh).sum()
            assert (g.nsl > 0) == (not weighted and R % vec == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("R", [3, 4, 6, 16, 20])
def test_apply_without_light_rows(weighted, R):
    import torch
    import polar_b200 as pg
    n = 100
    E = np.stack(np.triu_indices(n, 1), 1)  # every row has 99 neighbours
    w = np.linspace(0.5, 2.0, len(E)) if weighted else None
    G = pg.Graph(n, E, 1e-2, weights=w, heavy_thresh=8)
    x = torch.randn((n, R), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(R))
    M = torch.as_tensor(np.asarray(G.M0.get().todense())).cuda()
    # rows of 100 terms: 100 roundings of |M| |x| at most
    bound = 100 * 2.0 ** -52 * (M.abs() @ x.abs())
    assert bool(((pg.Op(G)(x) - M @ x).abs() < bound).all())
