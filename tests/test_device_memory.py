"""The engines' idle workspaces never make a call fail: every device allocation of the library asks for them back when
the device has no room."""
import glob
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lapstack_b200", "csrc")


def test_every_device_allocation_goes_through_the_one_that_asks_for_room():
    calls = {}
    for p in glob.glob(os.path.join(CSRC, "*")):
        if p.endswith((".cu", ".cuh", ".h")):
            code = re.sub(r"//[^\n]*", "", open(p).read())
            n = len(re.findall(r"\bcudaMalloc(?:Async|Pitch|Managed|3D)?\s*\(", code))
            if n:
                calls[os.path.basename(p)] = n
    assert calls == {"lsb_api.cu": 2}  # lsb_dev_alloc's own two


MB = 1 << 20


def _planes(w, h):
    rng = np.random.default_rng(w)
    return [rng.random((h, w), dtype=np.float32) for _ in range(3)]


def _stack(eng, how):
    """A 1024 x 768 stack whose buffers are there; the allocations of its run are still to come."""
    import lapstack_b200 as L
    if how == "halo":
        return eng.stack(1024, 768, 12, L.FuseParams(levels=4, halo=2.0, depth_level=0), None, None, brightness=False, crop=False)
    return eng.stack(1024, 768, 12, None, None, L.DepthParams(scale=0) if how == "solve" else None, brightness=False, crop=False)


def _use(st, how, frames):
    for f in frames:
        if how == "planes":
            st.push_f32((f.astype(np.float32) / 65535).transpose(2, 0, 1).copy())
        else:
            st.push_u16(f)
    out = st.finish()
    return [out.image_u16.copy(), out.winner.copy()] + ([out.depth.depth.copy()] if out.depth is not None else [])


def _net(net):
    import torch
    x = torch.zeros((1, 384, 512, 32), dtype=torch.bfloat16, device="cuda")
    return [net.forward(x, torch.zeros((1, 384, 512), device="cuda")).cpu().numpy()]


# what a run allocates (MB): the solver of its 1024 x 768 depth grid 75; 12 frames of float planes 113; the halo weights
# 50; the network's activations 90; a resize from 25 Mpx 115
@pytest.mark.gpu
@pytest.mark.parametrize("how", ["solve", "planes", "halo", "network", "resize"])
@pytest.mark.parametrize("idle_in", ["its own engine", "another engine"])
def test_a_run_finds_room_while_workspaces_are_idle(how, idle_in):
    import lapstack_b200 as L
    import torch
    eng = L.Engine()
    keeper = eng if idle_in == "its own engine" else L.Engine()
    frames, _ = L.synth_stack(L.SynthSpec(1024, 768, 12, seed=4))
    src = _planes(6000, 4100)[0][None] if how == "resize" else None

    def make():
        return _stack(eng, how) if how in ("solve", "planes", "halo") else L.UNet(seed=1) if how == "network" else None

    def use(obj):
        if how == "resize":
            return [eng.resize(src, 700, 500)]
        return _net(obj) if how == "network" else _use(obj, how, frames)

    first = make()
    want = use(first)  # also loads every kernel
    if first is not None:
        first.close()
    obj = make()
    d, c, g = _planes(3000, 2000)
    a = L.wls_solve(d, c, g, 3.0, 0.04, max_iters=4, engine=keeper)[0]  # 670 MB, idle from here on
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    x = torch.zeros((1, 384, 512, 32), dtype=torch.bfloat16, device="cuda") if how == "network" else None
    del x  # stays in torch's own cache
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - 36 * MB, dtype=torch.uint8, device="cuda")
    try:
        got = use(obj)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert all(np.array_equal(p, q) for p, q in zip(got, want))
    b = L.wls_solve(d, c, g, 3.0, 0.04, max_iters=4, engine=keeper)[0]  # made again
    assert np.array_equal(a, b)
    if obj is not None:
        obj.close()
    for e in {id(eng): eng, id(keeper): keeper}.values():
        e.close()
