"""Standalone calls (the WLS solve, the depth pass over given slices, a registered pair) keep their workspaces in the
engine: a call that finds one gives what a first call on a new engine gives, whatever sizes and settings came between
and whether its arrays are pageable, page-locked or too small to be staged; an error leaves the engine usable."""
import threading

import numpy as np
import pytest

import lapstack_b200 as L

pytestmark = pytest.mark.gpu


def _planes(w, h, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    guide = (0.5 + 0.3 * np.sin(x / 17.0) * np.cos(y / 11.0) + 0.02 * rng.standard_normal((h, w))).astype(np.float32)
    d = (5 + 3 * np.cos(x / 40.0) + 0.4 * rng.standard_normal((h, w))).astype(np.float32)
    return d, rng.random((h, w), dtype=np.float32), guide


def _calls(eng):
    """One of each kind at sizes below and above the staging threshold (1 MB a plane), odd ones among them."""
    out = []
    for w, h, em, vm in [(61, 47, 0, 0), (640, 513, 0, 0), (61, 47, 1, 1), (1201, 901, 1, 0), (640, 513, 0, 1)]:
        out.append(L.wls_solve(*_planes(w, h, w + h), 3.0 - 2.5 * em, 0.04, edge_mode=em, vcycle_mode=vm, engine=eng)[0])
    for w, h, n, kw in [(190, 131, 5, {}), (1280, 961, 6, {}), (190, 131, 5, dict(agg_radius=8, robust=0.0)),
                        (1280, 961, 6, dict(upsample="bilinear", median=False)), (190, 131, 5, dict(scale=2))]:
        p = L.DepthParams(**kw)
        k = 1 << p.scale
        rng = np.random.default_rng(n + w)
        sl = rng.random((n, (h + k - 1) // k, (w + k - 1) // k), dtype=np.float32)
        m = L.depth_from_slices(sl, np.stack(_planes(w, h, 9)[2:] * 3), p, engine=eng)
        out += [m.depth, m.conf, m.floor]
    for w, h in [(258, 172), (700, 525), (258, 172)]:
        f, _ = L.synth_stack(L.SynthSpec(w, h, 2, warp=True, mag_step=0.0, seed=w))
        sim, ev = L.multiscale_align(*(f[..., 1].astype(np.float32) / 65535), engine=eng)
        out += [sim, np.array(ev)]
    return out


def test_a_kept_workspace_gives_the_first_calls_results():
    fresh = []
    eng = L.Engine()
    fresh = _calls(eng)
    again = _calls(eng)  # every workspace found, or evicted and made again
    eng.close()
    other = L.Engine()
    _calls(other)[0]
    with pytest.raises(L.LsbError):
        L.depth_from_slices(np.zeros((2, 8, 8), np.float32), np.zeros((3, 16, 16), np.float32), L.DepthParams(agg_radius=60), engine=other)
    third = _calls(other)
    other.close()
    for a, b, c in zip(fresh, again, third):
        assert np.array_equal(a, b) and np.array_equal(a, c)


def test_pinned_and_pageable_arrays_agree():
    import torch
    eng = L.Engine()
    planes = _planes(1400, 1001, 3)
    pinned = [torch.from_numpy(p).pin_memory().numpy() for p in planes]
    a = L.wls_solve(*planes, 3.0, 0.04, engine=eng)[0]
    b = L.wls_solve(*pinned, 3.0, 0.04, engine=eng)[0]
    assert np.array_equal(a, b)
    frames, _ = L.synth_stack(L.SynthSpec(701, 525, 3, seed=5))
    outs = []
    for conv in (lambda f: f, lambda f: torch.from_numpy(f.view(np.int16)).pin_memory().numpy().view(np.uint16),
                 lambda f: torch.from_numpy(f.view(np.int16)).cuda()):
        st = eng.stack(701, 525, 3, depth=L.DepthParams())
        for f in frames:
            st.push_u16(conv(f))
        outs.append(st.finish())
        st.close()
    for o in outs[1:]:
        assert np.array_equal(o.image_u16, outs[0].image_u16) and np.array_equal(o.depth.depth, outs[0].depth.depth)
    eng.close()


def test_threads_with_engines_of_their_own():
    engines = [L.Engine(), L.Engine()]
    ref = L.wls_solve(*_planes(900, 701, 1), 3.0, 0.04, engine=engines[0])[0]
    got = [[], []]

    def work(i):
        for _ in range(4):
            got[i].append(L.wls_solve(*_planes(900, 701, 1), 3.0, 0.04, engine=engines[i])[0])

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert all(np.array_equal(ref, g) for gs in got for g in gs) and len(got[0]) == len(got[1]) == 4
    [e.close() for e in engines]
