"""The maintenance update at the ends of its range, against NumPy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _maintain(X, Y, U, win, G, es, h, t):
    """polar_maintain on copies of NumPy arrays: the new X, Y, h, t."""
    import torch
    from polar_b200 import _lib
    lib = _lib.load()
    p, nA, q = X.shape
    f32 = [int(v.dtype == np.float32) for v in (X, U)]
    d = [torch.as_tensor(v.copy()).cuda() for v in (X, Y, U, win, G, es, h, t)]
    Xd, Yd, Ud, wd, Gd, ed, hd, td = d
    tmp = torch.empty(lib.polar_maintain_tmp_bytes(p, nA, q), dtype=torch.uint8, device="cuda")
    _lib.check(lib.polar_maintain(Xd.data_ptr(), q, Yd.data_ptr(), q, f32[0], p, nA, q, Ud.data_ptr(), f32[1], U.shape[2],
                                  wd.data_ptr(), Gd.data_ptr(), ed.data_ptr(), len(es), hd.data_ptr(), td.data_ptr(),
                                  tmp.data_ptr(), 0), "maintain")
    torch.cuda.synchronize()
    return [v.cpu().numpy() for v in (Xd, Yd, hd, td)]


def _win(col, a, b, e):
    win = np.zeros(6, np.int32)
    win[:3] = col, a, b
    win[4:] = np.array([e], np.int64).view(np.int32)
    return win


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("ua,ub", [(1e308, -1e308), (1e308, 0.0), (-1e308, 0.0), (3e-308, 0.0), (-1.0 + 2.0 ** -53, 0.0), (-1.0, 0.0)])
def test_update_divides_by_any_denominator(prec, ua, ub):
    """X -= u xi / D and Y += u eta / D with D = 1 + u_a - u_b infinite, huge, tiny or zero: the
    quotient u / D is the division's, 0, infinite or not a number where that one is."""
    p, nA, q = 2, 40, 8
    rng = np.random.default_rng(3)
    dt = np.float32 if prec == "mixed" else np.float64
    X, Y = (rng.normal(size=(p, nA, q)).astype(dt) for _ in range(2))
    U = rng.normal(size=(p, nA, 1)) * 10.0 ** rng.integers(-300, 300, (p, nA, 1))
    a, b, e = 0, nA - 1, 1
    U[:, a, 0], U[:, b, 0] = ua, ub
    G = rng.normal(size=(3, q))
    es = np.array([[0, nA - 1], [1, 2], [3, 4]], np.int32)
    h, t = rng.uniform(0.0, 1.0, (2, p, 3))
    Xn, Yn, _, _ = _maintain(X, Y, U, _win(0, a, b, e), G, es, h, t)
    with np.errstate(all="ignore"):
        for j in range(p):
            x, y, u = X[j].astype(np.float64), Y[j].astype(np.float64), U[j, :, 0]
            xi, eta, D = x[a] - x[b], G[e] - (y[a] - y[b]), 1.0 + u[a] - u[b]
            ud = u / D
            for got, want in ((Xn[j], x - np.outer(ud, xi)), (Yn[j], y + np.outer(ud, eta))):
                # product and sum in one rounding here, two in NumPy, then the bank's own
                size = np.maximum(np.abs(want), 1.0)
                np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
                big = ~np.isfinite(want.astype(dt)) | ~np.isfinite(got)
                np.testing.assert_array_equal(got[big], want.astype(dt)[big])
                err = np.abs(got.astype(np.float64) - want)[~big] / size[~big]
                assert err.size == 0 or err.max() < (2.0 ** -22 if prec == "mixed" else 2.0 ** -50)


def test_more_poles_than_a_grid_dimension():
    p, nA, q = 65537, 3, 2
    rng = np.random.default_rng(1)
    X, Y = rng.normal(size=(2, p, nA, q))
    U = rng.uniform(-0.2, 0.2, (p, nA, 1))
    G = rng.normal(size=(1, q))
    h, t = rng.uniform(0.0, 1.0, (2, p, 1))
    Xn, Yn, hn, tn = _maintain(X, Y, U, _win(0, 0, 2, 0), G, np.array([[1, 2]], np.int32), h, t)
    u = U[:, :, 0]
    xi, eta = X[:, 0] - X[:, 2], G - (Y[:, 0] - Y[:, 2])
    ud = u / (1.0 + u[:, :1] - u[:, 2:])
    cc = ud[:, 1] - ud[:, 2]
    for got, want in ((Xn, X - ud[:, :, None] * xi[:, None]), (Yn, Y + ud[:, :, None] * eta[:, None]),
                      (hn[:, 0], np.maximum(0, h[:, 0] - 2 * cc * ((X[:, 1] - X[:, 2]) * xi).sum(1) + cc * cc * (xi * xi).sum(1))),
                      (tn[:, 0], np.maximum(0, t[:, 0] + 2 * cc * ((Y[:, 1] - Y[:, 2]) * eta).sum(1) + cc * cc * (eta * eta).sum(1)))):
        # a dozen roundings of terms of at most a few hundred
        np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-12)
