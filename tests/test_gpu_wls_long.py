"""The start's sweeps along lines too long for the partition in shared memory: some 18,700 cells where the line is
weighted (the first sweep's rows), 28,000 where it is not. They take the partition through global memory."""
import numpy as np
import pytest

import lapstack_b200 as L
from test_gpu_wls_start import _start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(20001, 3), (29001, 35), (3, 29001), (33, 28803)])
def test_long_lines_match_f64(size):
    w, h = size
    rng = np.random.default_rng(w + h)
    y, x = np.mgrid[0:h, 0:w]
    g = (0.5 + 0.3 * np.sin(x / 9.0) * np.cos(y / 7.0) + 0.05 * rng.standard_normal((h, w))).astype(np.float32)
    d = (10 + 5 * np.sin((x + y) / 31.0) + rng.standard_normal((h, w))).astype(np.float32)
    conf = (0.5 + 0.5 * rng.random((h, w))).astype(np.float32)
    u, _, iters, _ = L.wls_solve(d, conf, g, 3.0, 0.04, max_iters=0, engine=L.default_engine())
    assert iters == 0
    ref = _start(d, conf, g, 3.0, 0.04)
    # The first sweep's weights are at least 1/2 and its lambda 1.15, the later ones' weights 1 and lambda below that: a
    # line's condition number is at most 1 + 4 x 2.3 < 10.2, and a cell takes part in at most 25 roundings
    assert np.abs(u - ref).max() <= 2.0 ** -24 * 64 * float(np.abs(d).max()) * 4, np.abs(u - ref).max()
