"""More kinds and sizes of standalone calls than an engine keeps workspaces for (8), and calls that fail with one in
hand: the ones thrown out are made again, nothing of a failed call is kept, and every result is a new engine's."""
import numpy as np
import pytest

import lapstack_b200 as L

pytestmark = pytest.mark.gpu


def _planes(w, h):
    rng = np.random.default_rng(w * 1000 + h)
    return [rng.random((h, w), dtype=np.float32) for _ in range(3)]


def _solve(eng, i):
    return L.wls_solve(*_planes(64 + 9 * i, 48 + 7 * i), 3.0, 0.04, engine=eng)[0]


def test_workspaces_thrown_out_are_made_again():
    fresh = L.Engine()
    want = [_solve(fresh, i) for i in range(11)]
    fresh.close()
    eng = L.Engine()
    for order in (range(11), (0, 10, 1, 9, 2, 8), range(10, -1, -1)):  # 0 to 2 are out after the first round
        for i in order:
            assert np.array_equal(_solve(eng, i), want[i]), i
    eng.close()


def test_a_call_that_is_refused_with_a_workspace_in_hand():
    eng = L.Engine()
    want = _solve(eng, 1)
    for _ in range(2):
        with pytest.raises(L.LsbError, match="65535"):
            L.depth_from_slices(np.zeros((2, 1, 35000), np.float32), np.zeros((3, 1, 70000), np.float32), L.DepthParams(), engine=eng)
    assert np.array_equal(_solve(eng, 1), want)
    eng.close()


def test_a_call_that_finds_no_room_at_all():
    import torch
    eng = L.Engine()
    want = _solve(eng, 2)
    big = _planes(3000, 2000)
    sol = L.wls_solve(*big, 3.0, 0.04, max_iters=4, engine=eng)[0]
    eng.close()
    eng = L.Engine()
    assert np.array_equal(_solve(eng, 2), want)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
    try:  # its planes fit, its solver does not, with nothing idle left to free
        with pytest.raises(L.LsbError, match="out of memory"):
            L.wls_solve(*big, 3.0, 0.04, max_iters=4, engine=eng)
        assert np.array_equal(_solve(eng, 2), want)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(L.wls_solve(*big, 3.0, 0.04, max_iters=4, engine=eng)[0], sol)
    eng.close()
