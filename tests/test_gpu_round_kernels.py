"""Scoring with the stable top-B and the maintenance kernels at their edges, against NumPy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,B,p,obj", [(1, 1, 1, 0), (255, 64, 3, 0), (256, 1, 8, 0), (257, 16, 9, 2), (1025, 64, 32, 0),
                                       (262145, 64, 2, 0), (700, 5, 1, 1), (300000, 16, 17, 2)])
@pytest.mark.parametrize("values", ["spread", "ties", "dead"])
def test_score_topb(N, B, p, obj, values):
    import torch
    from polar_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(N + B)
    h, t = rng.uniform(0.1, 2.0, (p, N)), rng.uniform(0.1, 2.0, (p, N))
    live = np.ones(N, np.uint8)
    if values == "ties":  # three score values
        k = rng.integers(0, 3, N)
        h, t = np.broadcast_to(0.5 + k, (p, N)).copy(), np.ones((p, N))
    if values == "dead":  # fewer live ones than B, and scores that are not numbers
        live[rng.permutation(N)[min(N, B // 2):]] = 0
        h[:, N // 2] = np.nan
    tau, om, sigma = rng.uniform(0.0, 3.0, p), rng.uniform(0.1, 1.0, p), 0.01
    if obj == 1:
        g = np.log1p(t[0] + sigma * h[0])
    else:
        g = np.zeros(N)
        for j in range(p):
            g += om[j] * h[j] if obj == 2 else om[j] * h[j] / (1.0 + t[j] + (sigma + tau[j]) * h[j])
    masked = np.where(live != 0, g, -np.inf)
    order = [i for i in np.argsort(-masked, kind="stable") if not np.isnan(masked[i])][:B]
    d = [torch.as_tensor(x).cuda() for x in (h, t, tau, om, live)]
    tmp = torch.empty(lib.polar_topb_tmp_bytes(N, B), dtype=torch.uint8, device="cuda")
    idx = torch.full((B,), -7, dtype=torch.int64, device="cuda")
    val, every = torch.empty(B, dtype=torch.float64, device="cuda"), torch.empty(N, dtype=torch.float64, device="cuda")
    for out in (None, every.data_ptr()):
        _lib.check(lib.polar_score_topb(*(x.data_ptr() for x in d[:4]), sigma, p, N, d[4].data_ptr(), obj, B,
                                        idx.data_ptr(), val.data_ptr(), out, tmp.data_ptr(), 0), "score")
        torch.cuda.synchronize()
        got = idx.cpu().numpy()[:len(order)]
        if obj == 1 and values == "spread":  # log1p may differ in the last place
            np.testing.assert_allclose(masked[got], masked[order], rtol=1e-14)
        else:
            assert got.tolist() == [int(i) for i in order]
        np.testing.assert_allclose(val.cpu().numpy()[:len(order)], masked[order], rtol=1e-14)
        assert (idx.cpu().numpy()[len(order):] == np.iinfo(np.int64).max).all()
    np.testing.assert_allclose(every.cpu().numpy(), g, rtol=1e-14)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("q,pad,nA", [(1, 0, 3), (7, 1, 512), (32, 0, 513), (44, 4, 31), (64, 0, 1030), (129, 0, 40),
                                      (520, 8, 33)])
def test_maintain(prec, q, pad, nA):
    import torch
    from polar_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(q)
    p, N, B = 3, 50, 2
    dt = np.float32 if prec == "mixed" else np.float64
    X, Y = (rng.normal(size=(p, nA, q + pad)).astype(dt) for _ in range(2))
    U = (0.1 * rng.normal(size=(p, nA, B))).astype(dt)
    es = np.stack([rng.integers(0, nA, N), rng.integers(0, nA, N)], 1).astype(np.int32)
    G = rng.normal(size=(N, q))
    h, t = rng.uniform(0.0, 1.0, (p, N)), rng.uniform(0.0, 1.0, (p, N))
    e, a, b, col = 5, 0, nA - 1, 1
    U[:, a, col], U[:, b, col] = 0.3, -0.2
    win = np.zeros(6, np.int32)
    win[:3] = col, a, b
    win[4:] = np.array([e], np.int64).view(np.int32)
    X2, Y2, h2, t2 = X.astype(np.float64), Y.astype(np.float64), h.copy(), t.copy()
    ea, eb = es[:, 0], es[:, 1]
    for j in range(p):
        x, y, u = X2[j, :, :q], Y2[j, :, :q], U[j, :, col].astype(np.float64)
        xi, eta, D = x[a] - x[b], G[e] - (y[a] - y[b]), 1.0 + u[a] - u[b]
        wx, wy, cc = x @ xi, y @ eta, (u[ea] - u[eb]) / D
        h2[j] = np.maximum(0, h2[j] - 2 * cc * (wx[ea] - wx[eb]) + cc * cc * (xi @ xi))
        t2[j] = np.maximum(0, t2[j] + 2 * cc * (wy[ea] - wy[eb]) + cc * cc * (eta @ eta))
        X2[j, :, :q], Y2[j, :, :q] = x - np.outer(u, xi / D), y + np.outer(u, eta / D)
    d = {k: torch.as_tensor(v.copy()).cuda() for k, v in dict(X=X, Y=Y, U=U, es=es, G=G, h=h, t=t, win=win).items()}
    f32 = 1 if prec == "mixed" else 0
    tmp = torch.empty(lib.polar_maintain_tmp_bytes(p, nA, q), dtype=torch.uint8, device="cuda")
    dh, dt_ = torch.empty_like(d["h"]), torch.empty_like(d["t"])
    for split in (True, False):  # the split form first, on copies of the banks
        Xd, Yd = (d["X"].clone(), d["Y"].clone()) if split else (d["X"], d["Y"])
        fn, hh, tt = (lib.polar_maintain_split, dh, dt_) if split else (lib.polar_maintain, d["h"], d["t"])
        _lib.check(fn(Xd.data_ptr(), q + pad, Yd.data_ptr(), q + pad, f32, p, nA, q, d["U"].data_ptr(), f32, B,
                      d["win"].data_ptr(), d["G"].data_ptr(), d["es"].data_ptr(), N, hh.data_ptr(), tt.data_ptr(),
                      tmp.data_ptr(), 0), "maintain")
        torch.cuda.synchronize()
        eps = 1.2e-7 if f32 else 1e-14  # one rounding of each entry
        np.testing.assert_allclose(Xd.cpu().numpy(), X2, rtol=eps, atol=eps)
        np.testing.assert_allclose(Yd.cpu().numpy(), Y2, rtol=eps, atol=4 * eps)
    # sums of q products of size about 1
    np.testing.assert_allclose(d["h"].cpu().numpy(), h2, rtol=1e-12, atol=1e-13 * q)
    np.testing.assert_allclose(d["t"].cpu().numpy(), t2, rtol=1e-12, atol=1e-13 * q)
    np.testing.assert_allclose(np.maximum(0, h + dh.cpu().numpy()), h2, rtol=1e-12, atol=1e-13 * q)
    np.testing.assert_allclose(np.maximum(0, t + dt_.cpu().numpy()), t2, rtol=1e-12, atol=1e-13 * q)
