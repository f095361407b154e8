"""Levels one row or one column thin, against the oracle, bit for bit (halo control: to
the last bits of its exponentials): reflect-101 then sends every row of the window
to row 0, an even one, whatever its own parity. Frames one row high or one column wide, and explicit level counts that
reduce a level to one."""
import numpy as np
import pytest

import lapstack_b200 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _same(a, b, what):
    bad = np.count_nonzero(a != b)
    assert bad == 0, f"{what}: {bad} of {a.size} differ"


@pytest.mark.parametrize("halo", [0.0, 1.5])
@pytest.mark.parametrize("radius", [1, 2])
@pytest.mark.parametrize("w,h,levels", [(331, 1, 0), (331, 1, 3), (1, 331, 3), (1, 1, 1), (130, 2, 2), (2, 130, 2), (257, 9, 6), (9, 257, 6),
                                        (120, 3, 3)])
def test_thin_levels_match_the_oracle(w, h, levels, radius, halo):
    rng = np.random.default_rng(100 * w + h + radius)
    # frames that differ by a few units in the last place: the selection hangs on the last bits of the energies
    base = rng.random((3, h, w), np.float32)
    if halo:
        frames = [rng.random((3, h, w), np.float32) for _ in range(4)]
    else:
        frames = [base * (1 + rng.integers(0, 4, base.shape).astype(np.float32) * np.float32(2.0 ** -23)) for _ in range(4)]
    p = L.FuseParams(energy_radius=radius, levels=levels, depth_level=0, halo=halo)
    ref = O.Fuser(w, h, O.FuseParams(**vars(p)))
    dev = L.GpuFuser(w, h, p, n_max=len(frames))
    for f in frames:
        ref.push(f)
        dev.push(f)
    ri, rw = ref.finish()
    di, dw = dev.finish()
    _same(rw, dw, "winner map")
    if halo == 0.0:
        _same(ri, di, "fused image")
    else:  # the halo weights are expf/logf of the energies: the oracle's and CUDA's differ by their last bits
        assert np.abs(ri - di).max() <= 1e-5
