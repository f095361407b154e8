"""The bounded wait of the device search running out where it would in use: behind the levels that one cluster has
searched. The pair's call reports it, and the engine's next one is right."""
import numpy as np
import pytest

import lapstack_b200 as L

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_behind_the_cluster_is_reported(monkeypatch):
    import torch
    from torch.profiler import ProfilerActivity, profile
    f, _ = L.synth_stack(L.SynthSpec(700, 525, 2, warp=True, mag_step=0.0, seed=3))
    pair = [p.astype(np.float32) / 65535 for p in f[..., 1]]
    eng = L.Engine()
    want = L.multiscale_align(*pair, engine=eng)
    monkeypatch.setenv("LSB_NM_SPIN_LIMIT", "1")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        with pytest.raises(L.LsbError):
            L.multiscale_align(*pair, engine=eng)
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if names:
        assert any("nm_cluster_kernel" in n for n in names) and any("nm_search_kernel" in n for n in names)
    monkeypatch.delenv("LSB_NM_SPIN_LIMIT")
    got = L.multiscale_align(*pair, engine=eng)
    eng.close()
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]
