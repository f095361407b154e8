"""The weight gradients' sums over many tiles, against f64: the output layer of a network that hands its input through,
so that both operands of the sums (the input's bf16 values and bf16(2 e / n)) are known exactly and all positive. A
tensor core's FP32 accumulator drops the bits below its last place, at each of a tile's 8 steps, so a sum that ran on
over a CTA's tiles would fall short in proportion to their number; taken out tile by tile it falls short by at most
(1 + 2 + ... + 8) / 8 units in the last place, 4.5 2^-23. The additions after that round to nearest, either way."""
import numpy as np
import pytest

from oracle import unet_ref as U

pytestmark = pytest.mark.gpu


def _hand_through():
    """Weights that bring input channel c % 3 to channel c of the output layer's input, and an output of 0."""
    offs, nw, nb = U.offsets()
    w, b = np.zeros(nw, np.float32), np.zeros(nb, np.float32)
    for i in (0, 1, 12, 13):
        c1, c2, co = U.LAYERS[i][2], U.LAYERS[i][5], U.LAYERS[i][6]
        wl = np.zeros((9, co, c1 + c2), np.float32)
        for o in range(co):
            wl[4, o, o % 3 if i == 0 else c1 + o if c2 else o] = 1.0
        w[offs[i][0]:offs[i][0] + wl.size] = wl.ravel()
    return w, b, offs[-1]


# tiles of 16 x 8 pixels over 148 CTAs: one each, a few, 55
@pytest.mark.parametrize("shape", [(1, 64, 128), (2, 160, 312), (1, 1024, 1024)])
def test_gradient_sums_do_not_fall_short_with_the_number_of_tiles(shape):
    import lapstack_b200 as L
    import torch
    B, H, W = shape
    n = B * H * W
    w, b, (wo, bo) = _hand_through()
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.zeros((B, H, W, 32), dtype=torch.bfloat16, device="cuda")
    x[..., :3] = (0.5 + 0.5 * torch.rand((B, H, W, 3), generator=g, device="cuda")).to(torch.bfloat16)
    tgt = -0.5 - torch.rand((B, H, W), generator=g, device="cuda")
    net = L.UNet(seed=0)
    net.set_params(w, b)
    net.train_step(x, torch.zeros_like(tgt), tgt, lr=0.0)
    gw, gb = net.grads()
    net.close()
    dz = (2 * -tgt / np.float32(n)).to(torch.bfloat16).double()
    pad = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    ref = torch.stack([(dz[..., None] * pad[:, ky:ky + H, kx:kx + W, :3]).sum((0, 1, 2)) for ky in range(3) for kx in range(3)]).cpu().numpy()
    got = gw[wo:wo + 9 * 32 * 32].reshape(9, 32, 32)[:, 0, :3].astype(np.float64)
    err = np.append((got / ref - 1).ravel(), gb[bo] / float(dz.sum()) - 1)
    print(shape, "mean", err.mean(), "largest", np.abs(err).max())
    assert abs(err.mean()) <= 5.5 * 2.0 ** -23
    assert np.abs(err).max() <= 12 * 2.0 ** -23
