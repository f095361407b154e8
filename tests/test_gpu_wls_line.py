"""The WLS solve of a grid one cell wide or high is the answer itself, not a start for the CG: the reference's Thomas
sweep (depth.rs:677 / :707) in its order, bit for bit, at lengths on both sides of those from which the start's sweeps
are partitioned. On a constant guide every edge weight is exactly 1, so numpy's float32 gives the same values."""
import numpy as np
import pytest

import lapstack_b200 as L

pytestmark = pytest.mark.gpu


def _line(n, seed):
    rng = np.random.default_rng(seed)
    d = (10 + 5 * np.sin(np.arange(n) / 31.0) + rng.standard_normal(n)).astype(np.float32)
    return d, (rng.random(n) ** 2).astype(np.float32)


def _solve(d, conf, w, h):
    g = np.full((h, w), 0.5, np.float32)
    return L.wls_solve(d.reshape(h, w), conf.reshape(h, w), g, 3.0, 0.04, engine=L.default_engine())[0].ravel()


def _thomas(d, conf, lam, F):
    """The sweep in arithmetic F over a line of n >= 2 cells whose edges are all 1."""
    n, lam, one = len(d), F(lam), F(1)
    wd = np.maximum(conf, 0).astype(np.float32) + np.float32(1e-4)
    c, r = np.zeros(n, F), np.zeros(n, F)
    for i in range(n):
        ap, ai, w = F(i > 0), F(i + 1 < n), F(wd[i])
        lower, upper = -lam * ap, -lam * ai
        m = (w + lam * (ap + ai)) - lower * (c[i - 1] if i else F(0))
        c[i] = upper / m
        r[i] = (w * F(d[i]) - lower * (r[i - 1] if i else F(0))) / m
    for i in range(n - 2, -1, -1):
        r[i] = r[i] - c[i] * r[i + 1]
    return r


@pytest.mark.parametrize("w,h", [(1, 2), (1, 63), (1, 64), (1, 65), (1, 1000), (1, 9001), (2, 1), (63, 1), (64, 1), (65, 1), (256, 1), (1000, 1),
                                 (9001, 1)])
def test_a_line_is_the_reference_sweep(w, h):
    d, conf = _line(w * h, w * 3 + h)
    assert np.array_equal(_solve(d, conf, w, h), _thomas(d, conf, 3.0, np.float32))
