"""lsb_config.grid_limit bounds the CTAs of the fold's level-0 kernel and of its selection, whatever the frame's size, and
changes no result: engines that share a GPU stay in their shares."""
import json

import numpy as np
import pytest

import lapstack_b200 as L

pytestmark = pytest.mark.gpu


def _grids(fn, path):
    """Kernel name -> the CTAs of each of its launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        out = fn()
        torch.cuda.synchronize()
    p.export_chrome_trace(str(path))
    grids = {}
    for e in json.load(open(path))["traceEvents"]:
        if e.get("cat") == "kernel":
            grids.setdefault(e["name"], []).append(int(np.prod(e["args"]["grid"])))
    return out, grids


# the fused level-0 kernel and the border's rectangles; the levels above in one launch; halo control's levels one by one
@pytest.mark.parametrize("limit,halo", [(7, 0.0), (100, 0.0), (7, 2.0)])
def test_the_selection_stays_within_the_grid_limit(limit, halo, tmp_path):
    w, h, n = 1203, 801, 5
    frames, _ = L.synth_stack(L.SynthSpec(w, h, n, seed=8))
    p = L.FuseParams(halo=halo, levels=4, depth_level=1 if halo else 0)

    def run(eng):
        st = eng.stack(w, h, n, p, None, None)
        for f in frames:
            st.push_u16(f)
        out = st.finish()
        st.close()
        return out

    whole = run(L.default_engine())
    eng = L.Engine(grid_limit=limit)
    run(eng)
    part, grids = _grids(lambda: run(eng), tmp_path / "trace.json")
    eng.close()
    if not grids:
        pytest.skip("no kernel records from the profiler")
    bounded = {k: v for k, v in grids.items() if "select_strip_kernel" in k or "fold0_kernel" in k}
    assert any("select_strip_kernel" in k for k in bounded)
    assert all(g <= limit for v in bounded.values() for g in v), bounded
    for a, b in ((whole.image_u16, part.image_u16), (whole.image, part.image), (whole.winner, part.winner), (whole.shares, part.shares)):
        assert np.array_equal(a, b)
