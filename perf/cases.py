"""The work users of this engine have it do, as cases that a timing program can run one by one.

Each family below is one public entry point with the inputs and handles a program holds before the
call. The sizes are the benchmark's workloads (bench.py's c1, c2, c3, c3s, its batch and its U-Net
training), cut in frame count where the full stack would not fit several times over, and odd sizes
of the same ranges. draw() spreads over the same families and ranges.

  stack    a whole focus stack: registration, gains, fold, collapse and the depth pass, with the
           results read back. "place" says where the frames are: "resident" (written into the stack's
           frame store, as a device decoder does), "device" (tensors that are pushed) or "pinned"
           (page-locked host frames that are pushed)
  fuser    the fuser contract: float32 planes pushed frame by frame, no registration, no depth
  slices   the depth pass alone on focus slices the caller has
  wls      the weighted-least-squares depth solve alone
  align    the registration of one luma plane onto another
  forward  the warm-start network's forward pass
  train    one training step of the network
"""
import math

import numpy as np
import torch

import lapstack_b200 as L
from lapstack_b200 import unet as U

_engines = {}


def _engine(storage):
    """One engine per storage mode, kept for the whole run as a program keeps it."""
    if storage not in _engines:
        _engines[storage] = L.Engine(device=0, storage=storage)
    return _engines[storage]


def _stack(name, w, h, n, storage, aligned, levels, radius, place, coarsen=3):
    return dict(name=name, kind="stack", w=w, h=h, n=n, storage=storage, aligned=aligned, coarsen=coarsen, levels=levels,
                radius=radius, place=place)


def listed():
    return [
        # the registration of a preview-sized pair, every level searched: all launches and hand-offs
        dict(name="align_516x344", kind="align", w=516, h=344, coarsen=0),
        # the benchmark's smallest stack: short kernels, the fixed costs of a run
        _stack("stack_1mp_f32", 1024, 768, 8, "f32", False, 6, 3, "resident"),
        # a small aligned stack of frames that are on the device already
        _stack("stack_3mp_aligned", 2048, 1536, 16, "unorm16", True, 0, 3, "device"),
        # decoded frames on the host, pushed one by one: copies, registration and fold side by side
        _stack("stack_24mp_aligned_pinned", 6000, 4000, 8, "unorm16", True, 0, 3, "pinned"),
        # the headline's frames, registration and storage, ten of its hundred frames
        _stack("stack_45mp_aligned", 8256, 5504, 10, "unorm16", True, 0, 3, "resident"),
        # the full-precision path with the wide guided filter, no registration (a tripod on a rail)
        _stack("stack_24mp_f32_r8", 6000, 4000, 8, "f32", False, 8, 8, "resident"),
        # float frames from a caller's own registration, odd sides
        dict(name="fuser_1501x999", kind="fuser", w=1501, h=999, n=6, levels=0),
        # a depth map again from kept slices (another lambda, another radius), odd sides
        dict(name="slices_2047x1365", kind="slices", w=2047, h=1365, n=20, radius=3),
        # the solve on the depth grid of a 12 MP frame, the reference's edge weights
        dict(name="wls_2120x1416", kind="wls", w=2120, h=1416, edge=0, vcycle=0),
        # the solve at full frame size with the large-grid settings
        dict(name="wls_4240x2832_bf16", kind="wls", w=4240, h=2832, edge=1, vcycle=1),
        # the network on the headline's grid
        dict(name="forward_2064x1376", kind="forward", b=1, w=2064, h=1376),
        # the training step of the benchmark: 8 crops of 256
        dict(name="train_8x256x256", kind="train", b=8, w=256, h=256),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _sides(rng, lo, hi):
    """Width and height of a frame with about _log(lo, hi) pixels, odd sides among them."""
    px, ratio = _log(rng, lo, hi), rng.uniform(1.2, 1.8)
    return int(math.sqrt(px * ratio)) + rng.randrange(2), int(math.sqrt(px / ratio)) + rng.randrange(2)


def draw(rng):
    kind = rng.choice(["stack", "stack", "stack", "fuser", "slices", "wls", "align", "forward", "train"])
    if kind == "stack":
        w, h = _sides(rng, 0.5e6, 40e6)
        n = max(4, min(rng.randrange(4, 25), int(250e6 / (w * h))))
        aligned = rng.random() < 0.6
        place = rng.choice(["resident", "device", "pinned"] if w * h * n < 120e6 else ["resident", "device"])
        c = _stack("", w, h, n, rng.choice(["f32", "unorm16", "unorm16", "f16"]), aligned, 0, rng.choice([3, 3, 8]), place,
                   rng.choice([1, 2, 3]))
        del c["name"]
        return c
    if kind == "fuser":
        w, h = _sides(rng, 0.3e6, 8e6)
        return dict(kind=kind, w=w, h=h, n=rng.randrange(3, 11), levels=rng.choice([0, 0, 5]))
    if kind == "slices":
        w, h = _sides(rng, 0.5e6, 8e6)
        return dict(kind=kind, w=w, h=h, n=rng.randrange(8, 33), radius=rng.choice([3, 3, 8]))
    if kind == "wls":
        w, h = _sides(rng, 0.2e6, 12e6)
        return dict(kind=kind, w=w, h=h, edge=rng.randrange(2), vcycle=rng.randrange(2))
    if kind == "align":
        w, h = _sides(rng, 0.1e6, 3e6)
        return dict(kind=kind, w=w, h=h, coarsen=rng.randrange(3))
    b = rng.choice([1, 1, 2]) if kind == "forward" else rng.randrange(2, 9)
    w, h = (_sides(rng, 0.1e6, 1.4e6) if kind == "forward" else _sides(rng, 0.01e6, 0.065e6))
    return dict(kind=kind, b=b, w=max(8, w // 8 * 8), h=max(8, h // 8 * 8))


# ------------------------------------------------------------------- inputs
class _Plane:
    """Device memory the engine owns, for torch.as_tensor."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _smooth(gen, h, w, cells, b=1):
    """Smooth random planes in [0, 1]: a bicubic surface through a coarse random grid."""
    g = torch.rand((b, 1, cells, cells), generator=gen, device="cuda")
    return torch.nn.functional.interpolate(g, size=(h, w), mode="bicubic", align_corners=True).clamp(0, 1)[:, 0]


def _scene(gen, h, w, b=1):
    """Scene planes in [0, 1]: surfaces, edges and fine texture."""
    t = torch.nn.functional.interpolate(torch.randn((b, 1, (h + 2) // 3, (w + 2) // 3), generator=gen, device="cuda"), size=(h, w),
                                        mode="bilinear")[:, 0]
    return (0.35 * _smooth(gen, h, w, 6, b) + 0.3 * (_smooth(gen, h, w, 14, b) > 0.5) + 0.15 + 0.06 * t).clamp(0, 1)


def _frames(w, h, n, warp, seed, st=None):
    """The engine's seeded synthetic stack, into st's frame store or as a CUDA tensor (n, h, w, 3) of 16-bit words."""
    spec = L.SynthSpec(w, h, n, seed=int(seed) + 1, warp=warp, mag_step=0.0 if warp else 0.002, noise_std=0.002)
    if st is not None:
        L.synth_stack_device(spec, st.frames_device(), st.e.stream)
        torch.cuda.synchronize()
        return torch.as_tensor(_Plane(st.frames_device(), (n, h, w, 3), "<i2"), device="cuda")
    t = torch.empty((n, h, w, 3), dtype=torch.int16, device="cuda")
    L.synth_stack_device(spec, t.data_ptr())
    torch.cuda.synchronize()
    return t


def _unit(frames):
    """16-bit words as float32 in [0, 1]."""
    return (frames.to(torch.int32) & 0xFFFF).float() / 65535.0


def _params(seed):
    """The network's parameters as its layers hold them: weights [tap][cout][cin] per layer, then biases."""
    g = torch.Generator(device="cpu").manual_seed(int(seed) % (1 << 62))
    ws, bs = [], []
    for i, (ci, co, _) in enumerate(U.CONVS):
        last = i + 1 == len(U.CONVS)
        w = torch.randn((9, co, ci), generator=g) * math.sqrt(2.0 / (9 * (3 if i == 0 else ci)))
        b = 0.05 * torch.randn(co, generator=g)
        if i == 0:
            w[:, :, 3:] = 0  # the input has three live channels
        if last:  # the output layer has one live channel, and starts near zero
            w *= 0.05
            w[:, 1:] = 0
            b[1:] = 0
        ws.append(w.reshape(-1))
        bs.append(b)
    return torch.cat(ws).numpy(), torch.cat(bs).numpy()


def _batch(case, seed):
    """The network's inputs and target for a batch: guide luma, raw depth, confidence; the solved depth."""
    g, b, h, w = _gen(seed), case["b"], case["h"], case["w"]
    depth = _smooth(g, h, w, 8, b)
    noise = torch.randn((b, h, w), generator=g, device="cuda")
    conf = (1.2 * _smooth(g, h, w, 20, b)) ** 2
    raw = (depth + 0.05 * noise * (1.3 - conf).clamp(min=0.05)).clamp(0, 1)
    x = torch.zeros((b, h, w, U.CH), dtype=torch.bfloat16, device="cuda")
    for c, plane in enumerate((_scene(g, h, w, b), raw, conf)):
        x[..., c] = plane.to(torch.bfloat16)
    return x, raw.contiguous(), depth.contiguous()


def _wls_planes(case, seed):
    g, h, w = _gen(seed), case["h"], case["w"]
    conf = (1.3 * _smooth(g, h, w, 24)[0]) ** 2
    d = 20.0 * _smooth(g, h, w, 7)[0] + 0.6 * torch.randn((h, w), generator=g, device="cuda") * (1.4 - conf).clamp(min=0.1)
    guide = _scene(g, h, w)[0]
    return [p.float().cpu().numpy() for p in (d, conf, guide)]


_WLS = {0: (3.0, 0.04), 1: (0.5, 0.02)}  # lambda and sigma_c of the two edge weights, as the benchmark runs them


def prepare(case, seed):
    kind = case["kind"]
    if kind == "stack":
        eng = _engine(case["storage"])
        align = L.AlignParams(coarsen=case["coarsen"]) if case["aligned"] else None
        st = eng.stack(case["w"], case["h"], case["n"], L.FuseParams(levels=case["levels"]), align,
                       L.DepthParams(agg_radius=case["radius"]))
        s = dict(kind=kind, st=st, n=case["n"], frames=None)
        if case["place"] == "resident":
            _frames(case["w"], case["h"], case["n"], case["aligned"], seed, st)
        else:
            t = _frames(case["w"], case["h"], case["n"], case["aligned"], seed)
            if case["place"] == "pinned":
                host = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
                host.copy_(t)
                s["host"] = host
                s["frames"] = list(host.numpy().view(np.uint16))
            else:
                s["frames"] = list(t)
        return s
    if kind == "fuser":
        eng = _engine("f32")
        st = eng.stack(case["w"], case["h"], case["n"], L.FuseParams(levels=case["levels"]), None, None, brightness=False, crop=False)
        f = _unit(_frames(case["w"], case["h"], case["n"], False, seed)).permute(0, 3, 1, 2).contiguous()
        return dict(kind=kind, st=st, n=case["n"], frames=list(f))
    if kind == "slices":
        g, n, h, w = _gen(seed), case["n"], case["h"], case["w"]
        fused = torch.stack([_scene(g, h, w)[0] for _ in range(3)])
        dh, dw = (h + 1) // 2, (w + 1) // 2
        z, tex = (n - 1) * _smooth(g, dh, dw, 7)[0], 0.02 + 0.2 * _smooth(g, dh, dw, 40)[0]
        k = torch.arange(n, device="cuda", dtype=torch.float32)[:, None, None]
        sl = tex * torch.exp(-0.5 * ((k - z) / 1.5) ** 2) + 0.004 * torch.rand((n, dh, dw), generator=g, device="cuda")
        return dict(kind=kind, eng=_engine("f32"), slices=sl.cpu().numpy(), fused=fused.cpu().numpy(),
                    params=L.DepthParams(agg_radius=case["radius"]))
    if kind == "wls":
        return dict(kind=kind, eng=_engine("f32"), planes=_wls_planes(case, seed), edge=case["edge"], vcycle=case["vcycle"])
    if kind == "align":
        f = _unit(_frames(case["w"], case["h"], 2, True, seed))
        y = f @ torch.tensor([0.2126, 0.7152, 0.0722], device="cuda")
        return dict(kind=kind, eng=_engine("f32"), planes=[p.cpu().numpy() for p in y], coarsen=case["coarsen"])
    net = U.UNet(device=0, seed=0)
    net.set_params(*_params(seed))
    x, d_in, target = _batch(case, seed)
    return dict(kind=kind, net=net, x=x, d_in=d_in, target=target)


# ------------------------------------------------------------------ the pass
def _result(o):
    r = dict(image=o.image, image_u16=o.image_u16, winner=o.winner, shares=o.shares, gains=o.gains, align=o.align, crop=list(o.crop))
    if o.depth is not None:
        r.update(depth=o.depth.depth, conf=o.depth.conf, floor=o.depth.floor)
    return r


def run(state):
    kind = state["kind"]
    if kind == "stack":
        st = state["st"]
        if state["frames"] is None:
            st.set_count(state["n"])
        else:
            st.set_count(0)
            for f in state["frames"]:
                st.push_u16(f)
        return _result(st.finish())
    if kind == "fuser":
        st = state["st"]
        st.set_count(0)
        for f in state["frames"]:
            st.push_f32(f)
        return _result(st.finish())
    if kind == "slices":
        m = L.depth_from_slices(state["slices"], state["fused"], state["params"], engine=state["eng"])
        return dict(depth=m.depth, conf=m.conf, floor=m.floor)
    if kind == "wls":
        lam, sigma = _WLS[state["edge"]]
        u, _, iters, _ = L.wls_solve(*state["planes"], lam, sigma, 200, edge_mode=state["edge"], vcycle_mode=state["vcycle"],
                                     engine=state["eng"])
        return dict(u=u, iters=int(iters))
    if kind == "align":
        sim, evals = L.multiscale_align(*state["planes"], coarsen=state["coarsen"], engine=state["eng"])
        return dict(sim=sim, evals=int(evals))
    net = state["net"]
    if kind == "forward":
        return dict(out=net.forward(state["x"], state["d_in"]))
    # the end of the cosine schedule: the whole step, with an update too small to move the weights,
    # so that every pass on one state is the same step
    loss = net.train_step(state["x"], state["d_in"], state["target"], 1e-10)
    gw, gb = net.grads()
    return dict(loss=float(loss), gw=gw, gb=gb)


# ---------------------------------------------------------------------- work
def work(case):
    k, w, h = case["kind"], case["w"], case["h"]
    px = w * h
    if k == "stack":
        # frames in; image (f32, u16), winner, depth and confidence out, the floor on the depth grid
        return dict(bytes=6 * px * case["n"] + px * (12 + 6 + 4 + 8 + 1), flops=0)
    if k == "fuser":
        return dict(bytes=12 * px * case["n"] + px * (12 + 6 + 4), flops=0)
    if k == "slices":
        return dict(bytes=px * case["n"] + px * (12 + 8 + 1), flops=0)
    if k == "wls":
        return dict(bytes=4 * 4 * px, flops=0)
    if k == "align":
        return dict(bytes=2 * 4 * px, flops=0)
    live = 0  # multiply-adds of the live channels: 3 inputs in the first layer, 1 output in the last
    for i, (ci, co, lv) in enumerate(U.CONVS):
        live += 9 * (3 if i == 0 else ci) * (1 if i + 1 == len(U.CONVS) else co) * (w >> lv) * (h >> lv) * case["b"]
    grid = px * case["b"]
    if k == "forward":
        return dict(bytes=grid * (6 + 4), flops=2 * live)
    return dict(bytes=grid * (6 + 4 + 4), flops=6 * live)


# --------------------------------------------------------------------- exact
def _exact_wls(case, seed):
    """(W + lambda L) u = W d in 64 bits: conjugate gradients with the diagonal as preconditioner, run to 1e-12."""
    lam, sigma = _WLS[case["edge"]]
    d, conf, g = (torch.from_numpy(p).cuda().double() for p in _wls_planes(case, seed))
    dx, dy = (g[:, :-1] - g[:, 1:]).abs(), (g[:-1] - g[1:]).abs()
    f = (lambda t: torch.exp(-t / sigma)) if case["edge"] == 0 else (lambda t: torch.exp(-t * t / (2 * sigma * sigma)))
    ex, ey, wd = lam * f(dx), lam * f(dy), conf.clamp(min=0) + 1e-4
    diag = wd.clone()
    diag[:, :-1] += ex
    diag[:, 1:] += ex
    diag[:-1] += ey
    diag[1:] += ey

    def apply(v):
        o = wd * v
        tx, ty = ex * (v[:, :-1] - v[:, 1:]), ey * (v[:-1] - v[1:])
        o[:, :-1] += tx
        o[:, 1:] -= tx
        o[:-1] += ty
        o[1:] -= ty
        return o

    b = wd * d
    u = d.clone()
    r = b - apply(u)
    z = r / diag
    p = z.clone()
    rz, stop = (r * z).sum(), 1e-12 * b.norm()
    for k in range(6000):
        ap = apply(p)
        a = rz / (p * ap).sum()
        u += a * p
        r -= a * ap
        if k % 50 == 0 and r.norm() < stop:
            break
        z = r / diag
        rz, old = (r * z).sum(), rz
        p = z + (rz / old) * p
    return u.cpu().numpy()


def _exact_net(case, seed):
    """The network in 64 bits on its bf16 weights and inputs: out0, and the loss and its gradients."""
    F = torch.nn.functional
    w, b = _params(seed)
    x, d_in, target = _batch(case, seed)
    train = case["kind"] == "train"
    W = torch.from_numpy(w).cuda().to(torch.bfloat16).double().requires_grad_(train)
    B = torch.from_numpy(b).cuda().double().requires_grad_(train)
    x = x.double().permute(0, 3, 1, 2)
    wo = bo = 0
    layers = []
    for ci, co, _ in U.CONVS:
        layers.append((W[wo:wo + 9 * co * ci].reshape(3, 3, co, ci).permute(2, 3, 0, 1), B[bo:bo + co]))
        wo, bo = wo + 9 * co * ci, bo + co

    def conv(i, t):
        wt, bias = layers[i]
        cols = []
        for j in range(t.shape[0]):  # one image at a time, as a product of its unfolded windows, in bands of rows
            pad, rows = F.pad(t[j:j + 1], (1, 1, 1, 1)), []
            step = max(1, (1 << 26) // (9 * t.shape[1] * t.shape[3]))
            for y in range(0, t.shape[2], step):
                band = pad[:, :, y:min(y + step, t.shape[2]) + 2]
                rows.append((wt.reshape(wt.shape[0], -1) @ F.unfold(band, 3)[0]).reshape(wt.shape[0], -1, t.shape[3]))
            cols.append(torch.cat(rows, 1))
        y = torch.stack(cols) + bias[:, None, None]
        return y if i + 1 == len(layers) else F.relu(y)

    up = lambda t: F.interpolate(t, scale_factor=2, mode="nearest")
    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, F.avg_pool2d(e0, 2)))
    e2 = conv(5, conv(4, F.avg_pool2d(e1, 2)))
    m = conv(7, conv(6, F.avg_pool2d(e2, 2)))
    m = conv(9, conv(8, torch.cat([up(m), e2], 1)))
    m = conv(11, conv(10, torch.cat([up(m), e1], 1)))
    m = conv(13, conv(12, torch.cat([up(m), e0], 1)))
    out = conv(14, m)[:, 0]
    if not train:
        return dict(out=out.cpu())
    loss = ((d_in.double() + out - target.double()) ** 2).mean()
    gw, gb = torch.autograd.grad(loss, [W, B])
    return dict(loss=float(loss), gw=gw.cpu(), gb=gb.cpu())


def exact(case, seed):
    """The solve and the network have values in 64 bits. The stacks, the depth pass and the search pick frames
    and simplex branches by comparing computed numbers, and pick others in 64 bits: they have none."""
    if case["kind"] == "wls":
        return dict(u=_exact_wls(case, seed), iters=None)
    if case["kind"] == "forward":
        with torch.no_grad():
            return _exact_net(case, seed)
    if case["kind"] == "train":
        return _exact_net(case, seed)
    return None
