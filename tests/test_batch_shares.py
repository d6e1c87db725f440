"""Grid shares of batched solves: the factor on the CPU, and solves whose shares add up to more
than the GPU on it."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from polar_b200.synth import chung_lu

ROOT = Path(__file__).resolve().parent.parent


def test_grid_factor(tmp_path):
    cases = [[0.1] * 8, [1.0, 0.5], [10.0, 0.3, 0.3, 0.3], [10.0] * 3, [0.9] * 4, [100.0, 1.5, 1.0, 0.2, 0.2],
             [0.26, 0.38, 0.54, 0.77, 1.09, 1.56, 2.2, 3.2], [5.0] * 64]
    src = tmp_path / "f.cc"
    src.write_text("#include <cstdio>\n#include \"batch_split.h\"\nint main() {\n" + "".join(
        'printf("%%.17g\\n", polar::grid_factor({%s}, 2.5, 0.25));\n' % ", ".join(map(str, c)) for c in cases) + "}\n")
    subprocess.check_call(["g++", "-std=c++17", "-I", str(ROOT / "polar_b200" / "csrc"), str(src), "-o", str(tmp_path / "f")])
    out = [float(x) for x in subprocess.check_output([str(tmp_path / "f")], text=True).split()]
    for c, f in zip(cases, out):
        asked = [sum(min(1.0, k * x) for x in c) for k in (0.25, f, 1.0)]
        if asked[2] <= 2.5:
            assert f == 1.0, c  # nothing shrinks that fits as it is
        elif asked[0] >= 2.5:
            assert abs(f - 0.25) < 1e-12, c
        else:
            assert abs(asked[1] - 2.5) < 1e-9, c
    assert out[2] == 1.0  # one large graph does not shrink three small ones


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(9000, 12000, 20000, 30000, 45000), (150000, 3000, 2500, 2000)])
def test_batch_above_its_shares(sizes):
    """Five graphs that ask for more than 2.5 GPUs, and one large with three small: each solve
    equals the single one (same arithmetic, another order of its sums)."""
    import polar_b200 as pg
    from polar_b200.batch import msolve_batch
    R, tau = 64, np.array([0.0, 0.5, 30.0])
    ops, Ws, acts = [], [], []
    for n in sizes:
        ops.append(pg.Op(pg.Graph(n, chung_lu(n, 6.0, 2.3, n, min_degree=1), 1e-1)))
        rng = np.random.default_rng(n)
        Ws.append(rng.normal(size=(n, R)))
        acts.append(np.sort(rng.permutation(n)[:500]))
    for prec, tol, bound in (("fp64", 1e-10, 1e-8), ("mixed", 1e-7, 1e-4)):
        res = msolve_batch(ops, Ws, [tau] * len(ops), acts, tol, track=True, precision=prec)
        for op, W, act, (X, h, it) in zip(ops, Ws, acts, res):
            Xs, hs, its = pg.msolve(op, W, tau, act, tol, track=True, precision=prec)
            assert float((X - Xs).double().norm() / Xs.double().norm()) < bound
            assert float(((h - hs).abs() / hs).max()) < bound
            assert np.abs(it - its).max() <= max(3, 0.15 * its.max())
