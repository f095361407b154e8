"""The sweeps that start the WLS solve (depth.rs:1022-1034: three separable sweeps, the first weighted by the
confidence), alone: with no CG iteration allowed the solve returns them. Held to the same sweeps in f64, line by line,
over lengths around the kernels' bounds: the one-thread sweep below 64, segment counts of 32, 64 and 128 and lengths
that leave segments partly or wholly past the end, columns in groups of 8 and, where 8 do not fit, fewer."""
import numpy as np
import pytest

import lapstack_b200 as L

pytestmark = pytest.mark.gpu


def _lines(f, wd, a, lam):
    """Thomas along axis 0 of (n, lines) f64 arrays: (wd + lam (a_{i-1} + a_i)) x_i - lam a_{i-1} x_{i-1} - lam a_i x_{i+1} = wd f."""
    n = f.shape[0]
    ap = np.vstack([np.zeros((1, f.shape[1])), a[:-1]])
    ai = a.copy()
    ai[-1] = 0.0
    diag, lo, up = wd + lam * (ap + ai), -lam * ap, -lam * ai
    c, d = np.zeros_like(f), np.zeros_like(f)
    for i in range(n):
        m = diag[i] - (lo[i] * c[i - 1] if i else 0.0)
        c[i] = up[i] / m
        d[i] = (wd[i] * f[i] - (lo[i] * d[i - 1] if i else 0.0)) / m
    x = d.copy()
    for i in range(n - 2, -1, -1):
        x[i] -= c[i] * x[i + 1]
    return x


def _start(d, conf, g, lam, sigma):
    d, conf, g = (p.astype(np.float64) for p in (d, conf, g))
    ex, ey = np.zeros_like(g), np.zeros_like(g)
    ex[:, :-1] = np.exp(-np.abs(g[:, :-1] - g[:, 1:]) / sigma)
    ey[:-1] = np.exp(-np.abs(g[:-1] - g[1:]) / sigma)
    u = d
    for t in (1, 2, 3):
        lt = 1.5 * lam * 4.0 ** (3 - t) / 63.0
        wd = np.maximum(conf, 0) + 1e-4 if t == 1 else np.ones_like(d)
        u = _lines(u.T, wd.T, ex.T, lt).T
        u = _lines(u, np.ones_like(d), ey, lt)
    return u


@pytest.mark.parametrize("size", [(63, 65), (64, 64), (257, 31), (256, 300), (258, 513), (1031, 129), (130, 1100), (2049, 67), (70, 3700), (9, 7100),
                                  (7300, 9), (66, 1), (1, 66)])
def test_start_sweeps_match_f64(size):
    w, h = size
    rng = np.random.default_rng(w * 7 + h)
    y, x = np.mgrid[0:h, 0:w]
    g = (0.5 + 0.3 * np.sin(x / 9.0) * np.cos(y / 7.0) + 0.05 * rng.standard_normal((h, w))).astype(np.float32)
    d = (10 + 5 * np.sin(x / 31.0) + rng.standard_normal((h, w))).astype(np.float32)
    conf = (rng.random((h, w)) ** 2).astype(np.float32)
    u, _, iters, _ = L.wls_solve(d, conf, g, 3.0, 0.04, max_iters=0, engine=L.engine.default_engine())
    assert iters == 0
    if min(w, h) == 1:  # one line: the direct solve
        f64 = [p.astype(np.float64).reshape(-1, 1) for p in (d, np.maximum(conf, 0) + np.float32(1e-4), g)]
        a = np.zeros_like(f64[2])
        a[:-1] = np.exp(-np.abs(f64[2][:-1] - f64[2][1:]) / 0.04)
        ref = _lines(f64[0], f64[1], a, 3.0).reshape(h, w)
    else:
        ref = _start(d, conf, g, 3.0, 0.04)
    # Diagonally dominant systems with non-negative inverses of unit row sums: a sweep's FP32 error is at most a few
    # roundings of its largest value per unknown that couples, up to lam / wd ~ 3e4 at the faintest cells of the first
    # weighted sweep (the direct solve: the same), and later sweeps average it.
    tol = 2.0 ** -24 * 64 * float(np.abs(d).max()) * (30 if min(w, h) == 1 else 4)
    assert np.abs(u - ref).max() <= tol, (np.abs(u - ref).max(), tol)
