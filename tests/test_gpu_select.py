"""The selection of a pyramid level in register strips, against the oracle:
tiles of 56 x 8 pixels, sides one short of, at and past them, levels smaller
than a window's reach, every window radius, frames that are shared out over
warps and frames that are not, and the border by reflection. The REDUCE and the
collapse run in strips of 30 and 60 columns under the same cases."""
import numpy as np
import pytest

import lapstack_b200 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _same(a, b, what):
    bad = np.count_nonzero(a != b)
    assert bad == 0, f"{what}: {bad} of {a.size} differ"


# 1 frame, 2 and 5 (groups of uneven size), 13 (more than the 6 warps of a CTA)
@pytest.mark.parametrize("radius", [0, 1, 2])
@pytest.mark.parametrize("w,h,n", [(8, 8, 2), (55, 9, 1), (56, 8, 13), (57, 47, 5), (61, 49, 2), (120, 33, 5), (337, 131, 13), (344, 130, 5)])
def test_selection_matches_the_oracle(w, h, n, radius):
    rng = np.random.default_rng(1000 * w + h)
    frames = [rng.random((3, h, w), np.float32) for _ in range(n)]
    p = L.FuseParams(energy_radius=radius, use_chroma=bool((w + radius) & 1), depth_level=0)
    ref = O.Fuser(w, h, O.FuseParams(**vars(p)))
    dev = L.GpuFuser(w, h, p, n_max=n)
    for f in frames:
        ref.push(f)
        dev.push(f)
    ri, rw = ref.finish()
    di, dw = dev.finish()
    _same(rw, dw, "winner map")
    _same(ri, di, "fused image")
