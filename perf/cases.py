"""Workloads of this framework, each through its public entry points.

Families (the "kind" of a case):

- route          one DEM on a FlowRouter: receivers -> lake reroute -> accumulation
- many           a sequence of DEMs from pinned host memory through FlowRouter.route_many
- flood          GraphFlood from a dry start on one grid (Flooder.run_graphflood)
- ragged         a packed batch of uneven tiles routed in one call (RaggedRouter.route)
- ragged_flood   GraphFlood on a packed batch of tiles (RaggedFlooder.run)
- unet           the gradients of one warm-start U-Net training step

listed() names the cases, draw() gives others of the same ranges.  DEMs come from the
package's documented recipe (spectral 1/f^2 surface plus Gaussian pits), made on the GPU.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

DEV = "cuda"


def listed():
    return [
        # a small catchment routed interactively: launches and latency
        dict(name="route_small", kind="route", nx=48, ny=33, mode="normal", relief=300.0, pits=3, lakes=True,
             weighted=False, exact_order=False),
        # plain routing of a tilted 512 x 512 DEM, all edges outlets, no lake rerouting
        dict(name="route_plain", kind="route", nx=512, ny=512, mode="normal", relief=500.0, pits=0, lakes=False,
             weighted=False, exact_order=False),
        # an odd-sized clip with rainfall weights, periodic north-south
        dict(name="route_odd", kind="route", nx=1001, ny=777, mode="periodic_NS", relief=500.0, pits=150, lakes=True,
             weighted=True, exact_order=False),
        # reference-order f32 discharge on a 2048 x 2048 DEM
        dict(name="route_ordered", kind="route", nx=2048, ny=2048, mode="normal", relief=1500.0, pits=500, lakes=True,
             weighted=True, exact_order=True),
        # the headline: 4096 x 4096 with 2000 pits, periodic east-west, weighted discharge
        dict(name="route_large", kind="route", nx=4096, ny=4096, mode="periodic_EW", relief=1500.0, pits=2000,
             lakes=True, weighted=True, exact_order=False),
        # a DEM archive streamed from the host
        dict(name="many_1536", kind="many", nx=1536, ny=1280, count=6, mode="periodic_EW", relief=1500.0, pits=250),
        # a small GraphFlood run (the default 10 iterations)
        dict(name="flood_small", kind="flood", nx=256, ny=192, mode="normal", pits=8, iters=10),
        # GraphFlood at its benchmark size
        dict(name="flood_2048", kind="flood", nx=2048, ny=2048, mode="normal", pits=500, iters=10),
        # a batch of small watersheds
        dict(name="ragged_small", kind="ragged", tiles=48, lo=32, hi=160, pits=10, layout=7, graph=False),
        # the 512-tile ragged benchmark batch, replayed from its graph
        dict(name="ragged_512", kind="ragged", tiles=512, lo=128, hi=1024, pits=200, layout=4, graph=True),
        # training-data generation: GraphFlood on many equal tiles
        dict(name="ragged_flood", kind="ragged_flood", tiles=256, lo=128, hi=128, pits=8, layout=0, iters=10),
        # a training step of the warm-start network at its usual batch
        dict(name="unet_train", kind="unet", batch=16, height=128, width=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["route", "route", "many", "flood", "ragged", "ragged_flood", "unet"])
    if kind in ("route", "many", "flood"):
        hi = {"route": 4096, "many": 1536, "flood": 2048}[kind]
        nx, ny = _log_int(rng, 33, hi), _log_int(rng, 33, hi)
        if rng.random() < 0.4:  # real rasters are often cut to multiples of a block
            nx, ny = max(32, nx // 32 * 32), max(32, ny // 32 * 32)
        c = dict(kind=kind, nx=nx, ny=ny, mode=rng.choice(["normal", "periodic_EW", "periodic_NS"]),
                 pits=max(1, nx * ny * rng.randint(1, 4) // 16384))
        if kind == "route":
            c.update(relief=float(rng.randint(100, 1500)), lakes=rng.random() < 0.8, weighted=rng.random() < 0.6,
                     exact_order=rng.random() < 0.3)
        elif kind == "many":
            c.update(relief=float(rng.randint(100, 1500)), count=rng.randint(2, 6))
        else:
            c.update(iters=rng.randint(5, 12))
        return c
    if kind == "ragged":
        lo = _log_int(rng, 24, 256)
        return dict(kind=kind, tiles=_log_int(rng, 8, 256), lo=lo, hi=_log_int(rng, lo, 1024), pits=rng.randint(2, 100),
                    layout=rng.randint(1, 1 << 20), graph=rng.random() < 0.4)
    if kind == "ragged_flood":
        lo = _log_int(rng, 32, 160)
        return dict(kind=kind, tiles=_log_int(rng, 8, 256), lo=lo, hi=rng.choice([lo, _log_int(rng, lo, 256)]),
                    pits=rng.randint(1, 12), layout=rng.randint(1, 1 << 20), iters=rng.randint(5, 12))
    return dict(kind="unet", batch=_log_int(rng, 1, 16), height=8 * _log_int(rng, 4, 16), width=8 * _log_int(rng, 4, 16))


# ---- inputs ----------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _dem(nx, ny, gen, relief, pits, tilt=0.0):
    """Spectral 1/f^2 surface in [0, relief] m minus Gaussian pits (depth U(1, 20) m,
    radius U(3, 30) cells at 4096), in float64, rounded once: (ny, nx) float32."""
    k = torch.sqrt(torch.fft.fftfreq(ny, device=DEV, dtype=torch.float64)[:, None] ** 2
                   + torch.fft.rfftfreq(nx, device=DEV, dtype=torch.float64)[None, :] ** 2)
    k[0, 0] = 1.0
    f = torch.fft.rfft2(torch.randn(ny, nx, device=DEV, dtype=torch.float64, generator=gen)) / (k * k)
    f[0, 0] = 0.0
    z = torch.fft.irfft2(f, s=(ny, nx))
    z = (z - z.min()) / (z.max() - z.min()) * relief
    if tilt:
        z += tilt * torch.arange(ny, device=DEV, dtype=torch.float64)[:, None]
    if pits:
        u = torch.rand(4, pits, 1, device=DEV, dtype=torch.float64, generator=gen)
        r = (3.0 + 27.0 * u[3]) * max(max(nx, ny) / 4096.0, 0.05)
        gx = torch.exp(-((torch.arange(nx, device=DEV) - u[0] * nx) / r) ** 2)
        gy = torch.exp(-((torch.arange(ny, device=DEV) - u[1] * ny) / r) ** 2)
        z -= ((1.0 + 19.0 * u[2]) * gy).T @ gx
    return z.float()


def _rain(n, gen):
    """Per-cell precipitation weights, lognormal(0, 0.5)."""
    return torch.exp(0.5 * torch.randn(n, device=DEV, generator=gen))


def _layout(case):
    """Shapes, modes and pit counts of a ragged batch (part of the case, not of the seed)."""
    rng = random.Random(case["layout"])
    shapes = [(_log_int(rng, case["lo"], case["hi"]), _log_int(rng, case["lo"], case["hi"]))
              for _ in range(case["tiles"])]
    flood = case["kind"] == "ragged_flood"
    modes = ["normal" if flood or rng.random() < 0.5 else "periodic_EW" for _ in shapes]
    return shapes, modes, [rng.randint(0, case["pits"]) for _ in shapes]


def _packed_dems(case, gen, relief):
    shapes, _, pits = _layout(case)
    return torch.cat([_dem(nx, ny, gen, relief, p).reshape(-1) for (ny, nx), p in zip(shapes, pits)])


# the U-Net's convolutions: (Cin, Cout, level)
_CONVS = [(8, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (128, 256, 3), (256, 256, 3),
          (384, 128, 2), (128, 128, 2), (192, 64, 1), (64, 64, 1), (96, 32, 0), (32, 32, 0), (32, 8, 0)]


def _unet_inputs(case, seed):
    """(parameters, NHWC bf16 inputs, target, weight); the parameters as UNet.state_dict
    holds them, per convolution Cout x 3 x 3 x Cin weights then Cout biases."""
    rng = np.random.default_rng(seed)
    parts = []
    for cin, cout, _ in _CONVS:
        parts += [rng.standard_normal(cout * 9 * cin) * math.sqrt(2.0 / (9 * cin)), 0.05 * rng.standard_normal(cout)]
    n = case["batch"] * case["height"] * case["width"]
    gen = _gen(seed)
    x = torch.randn(n, 8, device=DEV, generator=gen) * 0.7
    x[:, 6:] = 0
    target = torch.randn(n, device=DEV, generator=gen) - 4.0
    weight = 1.0 + torch.rand(n, device=DEV, generator=gen) * 10.0
    return np.concatenate(parts).astype(np.float32), x.bfloat16().reshape(-1), target, weight


# ---- the cases -------------------------------------------------------------------------


def prepare(case, seed):
    from pyfastflow_b200.flow import FlowRouter, RaggedRouter
    from pyfastflow_b200.graphflood import Flooder, RaggedFlooder
    from pyfastflow_b200.warmstart import UNet

    kind, gen = case["kind"], _gen(seed)
    s = dict(case=case)
    if kind == "route":
        nx, ny = case["nx"], case["ny"]
        s["z"] = _dem(nx, ny, gen, case["relief"], case["pits"], 0.0 if case["lakes"] else 0.15)
        s["w"] = _rain(nx * ny, gen) if case["weighted"] else None
        s["router"] = FlowRouter(nx, ny, 30.0, boundary_mode=case["mode"], lakeflow=case["lakes"])
    elif kind == "many":
        nx, ny, n = case["nx"], case["ny"], case["count"]
        s["dems"] = [_dem(nx, ny, gen, case["relief"], case["pits"]).cpu().pin_memory() for _ in range(n)]
        s["rain"] = [_rain(nx * ny, gen).cpu().pin_memory() for _ in range(n)]
        s["Q"] = [torch.empty(nx * ny, pin_memory=True) for _ in range(n)]
        s["counts"] = [torch.empty(nx * ny, dtype=torch.int32, pin_memory=True) for _ in range(n)]
        s["router"] = FlowRouter(nx, ny, 30.0, boundary_mode=case["mode"])
    elif kind == "flood":
        nx, ny = case["nx"], case["ny"]
        s["z"] = _dem(nx, ny, gen, 1500.0, case["pits"])
        s["dry"] = torch.zeros(nx * ny, device=DEV)
        s["router"] = FlowRouter(nx, ny, 10.0, boundary_mode=case["mode"])
        s["flooder"] = Flooder(s["router"], precipitation_rates=1e-5, manning=0.033)
    elif kind == "ragged":
        shapes, modes, _ = _layout(case)
        s["z"] = _packed_dems(case, gen, 500.0)
        s["router"] = RaggedRouter(shapes, 30.0, modes)
        s["router"].seed_weights(_rain(s["router"].total, gen))
    elif kind == "ragged_flood":
        shapes, modes, _ = _layout(case)
        s["z"] = _packed_dems(case, gen, 200.0)
        s["router"] = RaggedRouter(shapes, 10.0, modes)
        u = np.random.default_rng(seed).uniform(size=(2, len(shapes)))
        s["flooder"] = RaggedFlooder(s["router"], precipitation_rates=5e-6 + 4.5e-5 * u[0], manning=0.02 + 0.04 * u[1])
    elif kind == "unet":
        p, s["x"], s["target"], s["weight"] = _unet_inputs(case, seed)
        s["net"] = UNet()
        s["net"].load_state_dict({"p": p})
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    r = s.get("router")
    if kind == "route":
        r.set_z(s["z"])
        r.compute_receivers()
        if case["lakes"]:
            r.reroute_flow()
        if s["w"] is not None:
            r.accumulate_weighted_Q(s["w"], exact_order=case["exact_order"])
        else:
            r.accumulate_constant_Q(1.0, area=True, exact_order=case["exact_order"])
        return dict(receivers=r.receivers, gradient=r.gradient, Q=r.Q, counts=r.counts)
    if kind == "many":
        r.route_many(s["dems"], s["rain"], s["Q"], s["counts"])
        return dict(Q=s["Q"], counts=s["counts"])
    if kind == "flood":
        f = s["flooder"]
        r.set_z(s["z"])
        r.Q.zero_()
        f.set_h(s["dry"])
        f.run_graphflood(case["iters"])
        return dict(h=f.h, z=r.z, Q=r.Q)
    if kind == "ragged":
        r.set_z(s["z"])
        r.route(graph=case["graph"])
        return dict(receivers=r.receivers, gradient=r.gradient, Q=r.Q, counts=r.counts)
    if kind == "ragged_flood":
        f = s["flooder"]
        r.set_z(s["z"])
        r.Q.zero_()
        f.h.zero_()
        f.run(case["iters"], stop=None)
        return dict(h=f.h, z=r.z, Q=r.Q)
    net = s["net"]
    pred = net.forward(s["x"], case["batch"], case["height"], case["width"], check=False)
    loss, dpred = net.loss_grad(s["target"], s["weight"])
    net.backward(dpred)
    return dict(pred=pred, loss=loss, grad=net.g)


def work(case):
    """What one pass cannot do without: each input read once, each output written once."""
    kind = case["kind"]
    if kind == "route":  # z (and weights) in; receivers, gradient, Q, counts out
        return dict(bytes=case["nx"] * case["ny"] * (24 if case["weighted"] else 20))
    if kind == "many":  # z and weights in; Q and counts out
        return dict(bytes=case["nx"] * case["ny"] * case["count"] * 16)
    if kind == "flood":  # z, h, Q in and out
        return dict(bytes=case["nx"] * case["ny"] * 24)
    if kind in ("ragged", "ragged_flood"):
        return dict(bytes=sum(a * b for a, b in _layout(case)[0]) * 24)
    pixels = case["batch"] * case["height"] * case["width"]
    macs = sum(9 * cin * cout * pixels / 4 ** lev for cin, cout, lev in _CONVS)
    params = sum(9 * cin * cout + cout for cin, cout, _ in _CONVS)
    # forward, data gradient (not of the first convolution) and weight gradient
    return dict(bytes=pixels * (16 + 32 + 8) + params * 8, flops=2 * (3 * macs - 9 * 8 * 32 * pixels))


# ---- the same in 64 bits, in plain torch -------------------------------------------------


def _drops(z, mode):
    """z minus each neighbour (top, left, right, bottom), -inf where there is none."""
    ew, ns = mode == "periodic_EW", mode == "periodic_NS"
    out = []
    for dim, shift, wraps in ((0, 1, ns), (1, 1, ew), (1, -1, ew), (0, -1, ns)):
        d = z - torch.roll(z, shift, dim)
        if not wraps:
            d.select(dim, 0 if shift > 0 else -1).fill_(-math.inf)
        out.append(d)
    return torch.stack(out)


def _exact_route(case, seed):
    gen = _gen(seed)
    nx, ny, mode = case["nx"], case["ny"], case["mode"]
    z = _dem(nx, ny, gen, case["relief"], case["pits"], 0.0 if case["lakes"] else 0.15)
    grad = _drops(z.double(), mode).amax(0).clamp_min(0).reshape(-1) / 30.0
    if case["lakes"]:  # Q hangs on the rerouted receivers, whole numbers that have to be equal
        return dict(receivers=None, gradient=grad, Q=None, counts=None)
    # receivers are the first steepest slope in f32; upstream sums by pointer doubling
    n = nx * ny
    slope = _drops(z, mode) / torch.tensor(30.0, device=DEV)
    cell = torch.arange(n, device=DEV).reshape(ny, nx)
    rec, best = cell.clone(), torch.zeros_like(z)
    for k, (dim, shift) in enumerate(((0, 1), (1, 1), (1, -1), (0, -1))):
        better = slope[k] > best
        rec = torch.where(better, torch.roll(cell, shift, dim), rec)
        best = torch.where(better, slope[k], best)
    rec = rec.reshape(-1)
    w = _rain(n, gen).double() if case["weighted"] else torch.full((n,), 900.0, device=DEV, dtype=torch.float64)
    q = torch.cat([w, w.new_zeros(1)])
    p = torch.where(rec == cell.reshape(-1), n, rec)  # roots flow into a sink past the grid
    p = torch.cat([p, p.new_full((1,), n)])
    for _ in range(max(1, math.ceil(math.log2(n)))):
        q = q.index_add(0, p[:n], q[:n])
        q[n] = 0
        p = p[p]
    return dict(receivers=None, gradient=grad, Q=q[:n], counts=None)


def _exact_unet(case, seed):
    import torch.nn.functional as F

    b, hh, ww = case["batch"], case["height"], case["width"]
    flat, x, target, weight = _unet_inputs(case, seed)
    p = torch.from_numpy(flat).to(DEV).double().requires_grad_(True)
    at, k = 0, 0

    def conv(t):
        nonlocal at, k
        cin, cout, _ = _CONVS[k]
        k += 1
        w = p[at:at + cout * 9 * cin].reshape(cout, 3, 3, cin).permute(0, 3, 1, 2)
        bias = p[at + cout * 9 * cin:at + cout * 9 * cin + cout]
        at += cout * 9 * cin + cout
        y = F.conv2d(t, w, bias, padding=1)
        return y if k == len(_CONVS) else y.relu()

    def up(t):
        return F.interpolate(t, scale_factor=2, mode="nearest")

    t = x.double().reshape(b, hh, ww, 8).permute(0, 3, 1, 2)
    e0 = conv(conv(t))
    e1 = conv(conv(F.avg_pool2d(e0, 2)))
    e2 = conv(conv(F.avg_pool2d(e1, 2)))
    t = conv(conv(F.avg_pool2d(e2, 2)))
    t = conv(conv(torch.cat([up(t), e2], 1)))
    t = conv(conv(torch.cat([up(t), e1], 1)))
    t = conv(conv(torch.cat([up(t), e0], 1)))
    pred = conv(t).permute(0, 2, 3, 1).reshape(-1, 8)
    loss = (weight.double() * (pred[:, 0] - target.double()) ** 2).sum() / weight.double().sum()
    (grad,) = torch.autograd.grad(loss, p)
    return dict(pred=pred.detach().reshape(-1), loss=loss.detach().reshape(1), grad=grad)


def exact(case, seed):
    if case["kind"] == "route":
        return _exact_route(case, seed)
    if case["kind"] == "unet":
        return _exact_unet(case, seed)
    # the other families route on surfaces with lakes: their values hang on whole-number
    # receivers, and GraphFlood feeds its own surface back into them
    return None
