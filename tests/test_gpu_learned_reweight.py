"""The robust solve of a stack with a learned start goes on from the first solve's solution. It is the reweighted system
that it solves: where the reweighting changes the answer, it runs iterations until that system's own residual is below
1e-5, and its depth is the plain solve's, not the first solve's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [0.1, 0.02])  # in frames; the noise of this stack's raw depth is about 0.3
def test_a_reweighting_that_matters_is_solved(tau):
    import lapstack_b200 as L
    from lapstack_b200 import unet as U
    n, eng, net = 6, L.default_engine(), U.UNet(seed=0)

    def rows(robust):
        return U.compare_warm_start(net, 512, 384, n, seeds=(7001,), engine=eng, depth=L.DepthParams(robust=robust), repeats=1)[0]

    once, twice = rows(0.0), rows(tau)
    net.close()
    first, plain, learned = once["learned"]["depth"], twice["plain"], twice["learned"]
    assert plain["rel"] < 1e-5 and learned["rel"] < 1e-5
    assert plain["iters"] > 0 and learned["iters"] > 0
    same = 1e-3 * (n - 1)  # two solves of one system to 1e-5
    assert np.abs(learned["depth"] - plain["depth"]).max() <= same
    assert np.abs(learned["depth"] - first).max() > 4 * same
