"""The kernels' launch shapes and fast forms against the general ones, at the sizes where
the choice changes: the device-driven reroute (one block, several, four launches), the
tree accumulation in one launch and in several, batch teams of 1 to 8 blocks, the
mma.sync tiles by channel count, the 16-byte forms of the network's small ops, and the
exact quotients and the power inside and outside their ranges.  All comparisons are bit
for bit unless a tolerance is derived beside it."""
import ctypes as C

import numpy as np
import pytest

from pyfastflow_b200 import synthetic

pytestmark = pytest.mark.gpu


def surface(kind, nx, ny, seed):
    rng = np.random.default_rng(seed)
    if kind == "zeros":  # flats and ties of both zeros
        return rng.choice(np.array([-0.0, 0.0, 1.0, -1.0], np.float32), size=(ny, nx))
    if kind == "int":
        return rng.integers(0, 30, (ny, nx)).astype(np.float32)
    if kind == "high":  # above the invalid key's 1e8
        return (rng.random((ny, nx)) * 4e8).astype(np.float32)
    return synthetic.spectral_dem(nx, ny, seed, relief=300.0, npits=max(1, nx * ny // 500), pit_scale=0.1)


def codes_like(mode, nx, ny, seed):
    rng = np.random.default_rng(seed)
    c = np.ones((ny, nx), np.uint8)
    c[rng.random((ny, nx)) < 0.02] = 0
    c[0, :] = c[-1, :] = 3
    c[1:-1, 0] = c[1:-1, -1] = 9
    return c


# <= 8192 cells: one block; < 1024 per SM: several; 360,000: four launches (148 SMs)
@pytest.mark.parametrize("nx,ny", [(2, 2), (48, 33), (64, 32), (65, 127), (92, 90), (513, 130), (600, 601)])
@pytest.mark.parametrize("kind", ["zeros", "int", "spectral", "high"])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_device_reroute_matches_host_loop(cuda, nx, ny, kind, mode):
    torch = cuda
    from pyfastflow_b200 import _lib
    from pyfastflow_b200.flow import FlowRouter

    names = ["normal", "periodic_EW", "periodic_NS", "custom"]
    z = surface(kind, nx, ny, nx + ny)
    lib = _lib.load()
    out = []
    for device_loop in (1, 0):
        prev = lib.pff_reroute_use_graphs(device_loop)
        try:
            r = FlowRouter(nx, ny, 10.0, names[mode], boundaries=codes_like(mode, nx, ny, 5) if mode == 3 else None)
            r.set_z(z)
            r.compute_receivers()
            r.reroute_flow()
            torch.cuda.synchronize()
        finally:
            lib.pff_reroute_use_graphs(prev)
        out.append({k: getattr(r, k).cpu().numpy() for k in
                    ("receivers", "receivers_", "bid", "basin_saddle", "outlet", "basin_saddlenode", "is_border",
                     "tag", "tag_", "z_")} | {"n": np.array(r.last_n_outer)})
    for k in out[0]:
        a, b = out[0][k], out[1][k]
        if a.dtype == np.float32:
            a, b = a.view(np.uint32), b.view(np.uint32)
        assert np.array_equal(a, b), k


# tiles of one row or column; one launch (<= 4 tiles per SM) and several (35 x 35 tiles)
@pytest.mark.parametrize("nx,ny", [(2, 2), (33, 65), (32, 33), (97, 31), (300, 512), (1100, 1100)])
@pytest.mark.parametrize("weighted", [False, True])
def test_tree_accumulation_shapes(cuda, nx, ny, weighted):
    torch = cuda
    from pyfastflow_b200.flow import FlowRouter

    r = FlowRouter(nx, ny, 30.0)
    r.set_z(surface("spectral", nx, ny, 3))
    r.compute_receivers()
    r.reroute_flow()
    w = synthetic.lognormal_weights(nx * ny, 4) if weighted else np.ones(nx * ny, np.float32)
    if weighted:
        r.accumulate_weighted_Q(w)
    else:
        r.accumulate_constant_Q(1.0, area=False)
    torch.cuda.synchronize()
    rec = r.receivers.cpu().numpy().astype(np.int64)
    # the sums in f64 by pointer doubling
    n = nx * ny
    q = np.stack([np.append(w.astype(np.float64), 0.0), np.append(np.ones(n), 0.0)])
    p = np.append(np.where(rec == np.arange(n), n, rec), n)
    while (p[:n] != n).any():
        add = np.stack([np.bincount(p[:n], weights=v[:n], minlength=n + 1) for v in q])
        q += add
        q[:, n] = 0
        p = p[p]
    assert np.array_equal(r.get_counts().ravel(), q[1, :n].astype(np.uint32))
    # one rounding to f32 (2^-24) of the exact sum; the f64 sums are off by < 1e-10
    got = r.get_Q().ravel().astype(np.float64)
    assert (np.abs(got - q[0, :n]) <= q[0, :n] * (2.0 ** -24 + 1e-9)).all()


# teams of 8, 4, 2 and 1 blocks per tile (148 SMs)
@pytest.mark.parametrize("ntiles,side", [(3, 190), (16, 110), (40, 75), (160, 24)])
@pytest.mark.parametrize("mode", ["normal", "periodic_EW", "periodic_NS"])
def test_batch_teams_match_single_grids(cuda, ntiles, side, mode):
    torch = cuda
    from pyfastflow_b200.flow import FlowRouter, RaggedRouter

    shapes = [(side + k % 3, side - k % 5) for k in range(ntiles)]
    zs = [surface("int" if k % 2 else "spectral", nx, ny, k) for k, (ny, nx) in enumerate(shapes)]
    rr = RaggedRouter(shapes, 30.0, mode)
    rr.set_z(zs)
    rr.seed_constant(1.0, area=True)
    rr.route()
    for t in list(range(0, ntiles, max(1, ntiles // 4)))[:5]:
        ny, nx = shapes[t]
        f = FlowRouter(nx, ny, 30.0, mode)
        f.set_z(zs[t])
        f.compute_receivers()
        f.reroute_flow()
        f.accumulate_constant_Q(1.0, area=True, exact_order=True)
        torch.cuda.synchronize()
        assert np.array_equal(rr.get_receivers(t), f.get_receivers()), t
        assert np.array_equal(rr.get_counts(t), f.get_counts()), t
        assert np.array_equal(rr.get_Q(t).view(np.uint32), f.get_Q().view(np.uint32)), t


# a team of 4 by the number of tiles, and by their average of more than 65536 cells
@pytest.mark.parametrize("ntiles,side", [(16, 75), (40, 262)])
def test_batch_teams_of_four(cuda, ntiles, side):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    total = sum((side + k % 3) * (side - k % 5) for k in range(ntiles))
    team = batch_shape(0, total, ntiles, 1024, 1)[2]
    if sms == 148:
        assert team == 4
    test_batch_teams_match_single_grids(cuda, ntiles, side, "normal")


@pytest.mark.parametrize("ntiles", [1, 20, 160])  # 8 blocks, 1 block, two half-size blocks per SM
@pytest.mark.parametrize("mode", ["normal", "periodic_EW", "periodic_NS"])
def test_batch_graphflood_teams_match_flooder(cuda, ntiles, mode):
    torch = cuda
    from pyfastflow_b200.flow import FlowRouter, RaggedRouter
    from pyfastflow_b200.graphflood import Flooder, RaggedFlooder

    side = 140 if ntiles == 1 else 37
    z = surface("spectral", side + 5, side, 8)
    rr = RaggedRouter([z.shape] * ntiles, 10.0, mode)
    rr.set_z([z] * ntiles)
    fl = RaggedFlooder(rr, precipitation_rates=1e-5)
    fl.run(4, stop=None)
    r = FlowRouter(z.shape[1], z.shape[0], 10.0, mode)
    r.set_z(z)
    f = Flooder(r, precipitation_rates=1e-5)
    f.run_graphflood(4)
    torch.cuda.synchronize()
    for t in (0, ntiles - 1):
        assert np.array_equal(fl.get_h(t).view(np.uint32), f.get_h().view(np.uint32)), t
        assert np.array_equal(rr.get_Q(t).view(np.uint32), r.get_Q().view(np.uint32)), t


# batches of small tiles, by the threads of a block and the largest tile; a larger one beside them,
# tiles of two rows, custom boundaries, more tiles than blocks
@pytest.mark.parametrize("threads,ctas", [(1024, 1), (512, 2), (256, 4)])
@pytest.mark.parametrize("sides,ntiles", [((2, 9), 20), ((38, 43), 30), ((43, 44), 30), ((50, 60), 30), ((59, 61), 30),
                                          ((20, 74), 160), ((24, 75), 160), ((12, 50), 310), ((12, 52), 310)])
def test_batches_of_small_tiles(cuda, threads, ctas, sides, ntiles):
    """Against single grids, and every launch shape and the graph alike."""
    torch = cuda
    from pyfastflow_b200.flow import FlowRouter, RaggedRouter

    rng = np.random.default_rng(ntiles)
    shapes = [tuple(int(v) for v in rng.integers(sides[0], sides[1] + 1, 2)) for _ in range(ntiles)]
    shapes[0] = (sides[1], sides[1])
    names = ["normal", "periodic_EW", "periodic_NS", "custom"]
    modes = [names[k % 4] for k in range(ntiles)]
    codes = [codes_like(3, nx, ny, k) if k % 4 == 3 else None for k, (ny, nx) in enumerate(shapes)]
    kinds = ["int", "spectral", "zeros"]
    zs = [surface(kinds[k % 3] if min(shapes[k]) > 4 else "int", nx, ny, k) for k, (ny, nx) in enumerate(shapes)]
    rr = RaggedRouter(shapes, 30.0, modes, codes=codes)
    rr.threads, rr.ctas_per_sm = threads, ctas
    rr.set_z(zs)
    rr.seed_weights(synthetic.lognormal_weights(rr.total, 4))
    rr.route()
    got = [t.clone() for t in (rr.receivers, rr.gradient, rr.Q, rr.counts)]
    for graph in (True, True, False):
        rr.route(graph=graph)
        for a, b in zip(got, (rr.receivers, rr.gradient, rr.Q, rr.counts)):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    for t in [0] + list(range(1, ntiles, ntiles // 8)):
        ny, nx = shapes[t]
        f = FlowRouter(nx, ny, 30.0, modes[t], boundaries=codes[t])
        f.set_z(zs[t])
        f.compute_receivers()
        f.reroute_flow()
        f.accumulate_weighted_Q(rr._slice(rr.seed, t), exact_order=True)
        torch.cuda.synchronize()
        assert np.array_equal(rr.get_receivers(t), f.get_receivers()), t
        assert np.array_equal(rr.get_counts(t), f.get_counts()), t
        assert np.array_equal(rr.get_Q(t).view(np.uint32), f.get_Q().view(np.uint32)), t


def batch_shape(graphflood, total, ntiles, threads, ctas):
    from pyfastflow_b200 import _lib

    v = [C.c_int(threads), C.c_int(ctas), C.c_int()]
    _lib.call("pff_batch_shape", graphflood, total, ntiles, *map(C.byref, v))
    return tuple(x.value for x in v)


def test_batch_graphflood_takes_the_shape_asked_for(cuda):
    """More tiles than SMs change only a shape that is left to the library."""
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    for n in (sms, sms + 1):
        for threads, ctas in ((1024, 1), (512, 1), (512, 2), (256, 2)):
            assert batch_shape(1, 1000 * n, n, threads, ctas)[:2] == (threads, ctas)
    assert batch_shape(1, 1000 * sms, sms, 1024, 0)[:2] == (1024, 1)
    assert batch_shape(1, 1000 * (sms + 1), sms + 1, 1024, 0)[:2] == (512, 2)
    assert batch_shape(1, 1000 * (sms + 1), sms + 1, 512, 0)[:2] == (512, 1)


@pytest.mark.parametrize("scale", [1e-37, 1e-20, 1e-9, 1.0, 1e9, 1e25, 1e36])
def test_diffusion_quotients_in_and_out_of_range(cuda, scale):
    """Mode 0's fused pass (Markstein quotients) against mode 3 with the same boundary
    (per-sweep kernels, IEEE divisions)."""
    torch = cuda
    from pyfastflow_b200 import _dev, _lib

    lib = _lib.load()
    nx, ny = 150, 90
    rng = np.random.default_rng(2)
    z = (rng.standard_normal((ny, nx)) * scale).astype(np.float32)
    z[rng.random((ny, nx)) < 0.1] *= np.float32(1e-18)  # neighbouring drops far apart
    z[5, 5] = np.nan
    codes = np.ones((ny, nx), np.uint8)
    codes[0, :] = codes[-1, :] = codes[:, 0] = codes[:, -1] = 3
    cd = torch.from_numpy(codes.ravel()).cuda()
    res = []
    for mode in (0, 3):
        zd = torch.from_numpy(z.ravel().copy()).cuda()
        Q = torch.full((nx * ny,), 2.5, device="cuda")
        tmp = torch.zeros(nx * ny, device="cuda")
        nb = lib.pff_diffuse_workspace_bytes(nx * ny)
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        _lib.call("pff_diffuse_q", zd.data_ptr(), Q.data_ptr(), tmp.data_ptr(), 5, nx, ny, 10.0, 1e-3, mode,
                  cd.data_ptr() if mode == 3 else None, ws.data_ptr(), nb, _dev.stream())
        q = Q.cpu().numpy()
        bits = q.view(np.uint32).copy()
        bits[np.isnan(q)] = 0x7FC00000
        res.append(bits)
    assert np.array_equal(res[0], res[1])


# the range's ends, octaves inside it, subnormals, zero, infinity, NaN, negatives
@pytest.mark.parametrize("lo,hi", [(0x1C7F0000, 0x1C810000), (0x627F0000, 0x62810000), (0x3F000000, 0x40800000),
                                   (0x30000000, 0x30FFFFFF), (0x50000000, 0x50FFFFFF), (0, 0x00900000),
                                   (0x7F7F0000, 0x7FC10000), (0x80000000, 0x80010000), (0xBF7F0000, 0xBF810000)])
def test_pow53_is_the_double_power(cuda, lo, hi):
    from pyfastflow_b200 import _lib

    bad = C.c_longlong(-1)
    _lib.call("pff_pow53_selfcheck", lo, hi, C.byref(bad))
    assert bad.value == 0


def _bf(torch, *shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g).to(torch.bfloat16)


@pytest.mark.parametrize("cin,cout", [(8, 8), (8, 16), (32, 24), (32, 32), (96, 40), (24, 64), (40, 96)])
@pytest.mark.parametrize("B,H,W", [(3, 7, 5), (1, 24, 40)])
def test_conv_tiles_by_channel_count(cuda, cin, cout, B, H, W):
    """Forward and weight gradient on the mma.sync path, tiles of 16, 32 and 64 output
    channels, against torch in f64 on the same bf16 operands: f32 sums of K products are off
    by less than K 2^-24 times the sum of magnitudes."""
    torch = cuda
    import torch.nn.functional as F

    from pyfastflow_b200 import _dev, _lib

    x, dy = _bf(torch, B, H, W, cin, seed=1).cuda(), _bf(torch, B, H, W, cout, seed=2).cuda()
    w = _bf(torch, cout, 9, cin, seed=3).cuda()
    y = torch.empty(B, H, W, cout, device="cuda")
    dw = torch.zeros(cout, 9, cin, device="cuda")
    prev = 0
    _lib.call("pff_conv_set_path", 1)
    try:
        _lib.call("pff_conv3x3_fwd", x.data_ptr(), cin, 0, w.data_ptr(), None, y.data_ptr(), cout, 0, B, H, W, cin, cout,
                  0, 1, _dev.stream())
    finally:
        _lib.call("pff_conv_set_path", prev)
    _lib.call("pff_conv3x3_wgrad", x.data_ptr(), cin, 0, dy.data_ptr(), cout, 0, dw.data_ptr(), B, H, W, cin, cout,
              _dev.stream())

    def f64(xd, wd, dyd):
        xt = xd.double().permute(0, 3, 1, 2)
        wt = wd.double().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2).clone().requires_grad_(True)
        o = F.conv2d(xt, wt, padding=1)
        (o * dyd.double().permute(0, 3, 1, 2)).sum().backward()
        return o.detach().permute(0, 2, 3, 1), wt.grad.permute(0, 2, 3, 1).reshape(cout, 9, cin)

    ry, rw = f64(x, w, dy)
    my, mw = f64(x.abs(), w.abs(), dy.abs())
    assert ((y.double() - ry).abs() <= 9 * cin * 2.0 ** -24 * my + 1e-30).all()
    assert ((dw.double() - rw).abs() <= B * H * W * 2.0 ** -24 * mw + 1e-30).all()


# channel blocks of 32 and 64 with and without padding; pixel tiles of 8 or 16 rows of 16 with remainders
@pytest.mark.parametrize("cin,cout", [(24, 24), (64, 32), (32, 64), (64, 64), (104, 72)])
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 8, 16), (3, 9, 17), (1, 15, 31), (2, 33, 40), (70, 8, 8)])
def test_weight_gradient_tiles(cuda, cin, cout, B, H, W):
    """The nine-tap weight gradient on channel slices, added onto dw, 4- and 8-byte aligned,
    against torch in f64 (tolerance as above).  An infinity in the last column reaches the
    same sums and no others."""
    torch = cuda
    import torch.nn.functional as F

    from pyfastflow_b200 import _dev, _lib

    x, dy = _bf(torch, B, H, W, cin + 16, seed=1).cuda(), _bf(torch, B, H, W, cout + 8, seed=2).cuda()
    n = cout * 9 * cin
    for inf, off in ((False, 0), (False, 1), (True, 0)):
        if inf:
            x[0, 0, W - 1, 8] = float("inf")
        xs, ds = x[..., 8:8 + cin].double(), dy[..., 8:].double()
        buf = torch.full((n + 1,), 0.5, device="cuda")
        dw = buf[off:off + n]
        _lib.call("pff_conv3x3_wgrad", x.data_ptr(), cin + 16, 8, dy.data_ptr(), cout + 8, 8, dw.data_ptr(), B, H, W, cin,
                  cout, _dev.stream())
        got = dw.double().reshape(cout, 9, cin)

        def ref(u, v):
            up = F.pad(u, (0, 0, 1, 1, 1, 1))
            taps = [torch.einsum("bhwo,bhwi->oi", v, up[:, t // 3:t // 3 + H, t % 3:t % 3 + W]) for t in range(9)]
            return torch.stack(taps, 1)

        fin = torch.where(torch.isfinite(xs), xs, torch.zeros((), dtype=torch.float64, device="cuda"))
        rw, mw = ref(fin, ds) + 0.5, ref(fin.abs(), ds.abs()) + 0.5
        hit = ref((~torch.isfinite(xs)).double(), ds.abs()) != 0
        assert torch.equal(~torch.isfinite(got), hit)
        assert ((got - rw).abs()[~hit] <= ((B * H * W + 150) * 2.0 ** -24 * mw + 1e-30)[~hit]).all()
        assert buf[n * (1 - off)].item() == 0.5


@pytest.mark.parametrize("cin", [8, 32, 64, 96])
@pytest.mark.parametrize("cout,f32", [(8, 0), (17, 1), (40, 0)])
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 16, 16), (1, 17, 18)])
def test_conv_tile_is_the_im2col_form(cuda, cin, cout, f32, B, H, W):
    """Tiles with a halo in shared memory against the im2col kernel, which a channel stride
    beyond 32-bit tile offsets takes: bit for bit, with an infinity in the last pixel."""
    torch = cuda
    from pyfastflow_b200 import _dev, _lib

    cs = (2 ** 31 // (20 * W + 32) + 8) // 8 * 8
    x = _bf(torch, B * H * W, cin, seed=1).cuda()
    x[-1, 3] = float("inf")
    w, bias = _bf(torch, cout, 9, cin, seed=3).cuda(), torch.linspace(-1, 1, cout, device="cuda")
    wide = torch.empty(B * H * W * cs, dtype=torch.bfloat16, device="cuda")
    wide.view(B * H * W, cs)[:, 16:16 + cin] = x
    out = []
    _lib.call("pff_conv_set_path", 1)
    try:
        for t, c, off in ((x, cin, 0), (wide, cs, 16)):
            y = torch.full((B * H * W, cout + 8), 7.0, device="cuda").to(torch.float32 if f32 else torch.bfloat16)
            _lib.call("pff_conv3x3_fwd", t.data_ptr(), c, off, w.data_ptr(), bias.data_ptr(), y.data_ptr(), cout + 8, 4,
                      B, H, W, cin, cout, 1, f32, _dev.stream())
            out.append(y)
    finally:
        _lib.call("pff_conv_set_path", 0)
    assert (out[0][:, :4] == 7).all() and (out[0][:, 4 + cout:] == 7).all() and (out[0][:, 4:4 + cout] == 0).any()
    dt = torch.int32 if f32 else torch.int16
    assert torch.equal(out[0].view(dt), out[1].view(dt))


def test_conv_tile_many_tiles(cuda):
    """More tiles than CTAs: two images' rows against each image by itself, bit for bit."""
    torch = cuda
    from pyfastflow_b200 import _dev, _lib

    B, H, W, cin, cout = 9, 120, 136, 32, 96
    x, w = _bf(torch, B, H, W, cin, seed=1).cuda(), _bf(torch, cout, 9, cin, seed=3).cuda()
    y, z = (torch.zeros(B, H, W, cout, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    _lib.call("pff_conv3x3_fwd", x.data_ptr(), cin, 0, w.data_ptr(), None, y.data_ptr(), cout, 0, B, H, W, cin, cout, 0, 0,
              _dev.stream())
    for b in range(B):
        _lib.call("pff_conv3x3_fwd", x[b].data_ptr(), cin, 0, w.data_ptr(), None, z[b].data_ptr(), cout, 0, 1, H, W, cin,
                  cout, 0, 0, _dev.stream())
    assert y.abs().sum() > 0 and torch.equal(y.view(torch.int16), z.view(torch.int16))


def test_weight_gradient_long_rows(cuda):
    """A channel stride beyond the tiles' 32-bit offsets takes the general kernel: the same
    gradient as for dense rows (tolerance as above, twice)."""
    torch = cuda
    from pyfastflow_b200 import _dev, _lib

    cs, cin, cout, W = 41_297_768, 24, 40, 3  # (20 W + 32) cs >= 2^31
    x, dy = _bf(torch, 1, 1, W, cin, seed=1).cuda(), _bf(torch, 1, 1, W, cout, seed=2).cuda()
    wide = torch.zeros(W * cs, dtype=torch.bfloat16, device="cuda")
    wide.view(W, cs)[:, 16:16 + cin] = x[0, 0]
    out = []
    for t, c, off in ((x, cin, 0), (wide, cs, 16)):
        dw = torch.zeros(cout, 9, cin, device="cuda")
        _lib.call("pff_conv3x3_wgrad", t.data_ptr(), c, off, dy.data_ptr(), cout, 0, dw.data_ptr(), 1, 1, W, cin, cout,
                  _dev.stream())
        out.append(dw)
    mag = dy.abs().float().amax() * x.abs().float().amax() * W
    assert out[0].abs().sum() > 0 and ((out[0] - out[1]).abs() <= 2 * W * 2.0 ** -24 * mag).all()


@pytest.mark.parametrize("C_,B,H,W", [(8, 1, 2, 2), (24, 3, 6, 10), (96, 2, 16, 8), (256, 1, 4, 6)])
def test_small_ops_16_byte_forms(cuda, C_, B, H, W):
    """Resampling and the ReLU / bias gradient on 8 channels per thread against the
    one-channel forms (taken for a slice at an offset that is no multiple of 8)."""
    torch = cuda
    from pyfastflow_b200 import _dev, _lib

    st = _dev.stream()

    def rows(t, off):  # the channels of t at offset off of rows 16 wider
        b = torch.zeros(t.shape[0], C_ + 16, dtype=torch.bfloat16, device="cuda")
        b[:, off:off + C_] = t
        return b

    fine, coarse = _bf(torch, B * H * W, C_, seed=1).cuda(), _bf(torch, B * H * W // 4, C_, seed=2).cuda()
    fine2 = _bf(torch, B * H * W, C_, seed=3).cuda()
    db = []
    res = []
    for off in (8, 4):
        f, c, acc = rows(fine, off), rows(coarse, off), rows(fine2, off)
        up, dn, ub = rows(fine * 0, off), rows(coarse * 0, off), rows(coarse * 0, off)
        cs = C_ + 16
        _lib.call("pff_avgpool2", f.data_ptr(), cs, off, dn.data_ptr(), cs, off, B, H, W, C_, st)
        _lib.call("pff_upsample2", c.data_ptr(), cs, off, up.data_ptr(), cs, off, B, H // 2, W // 2, C_, st)
        _lib.call("pff_upsample2_bwd", f.data_ptr(), cs, off, ub.data_ptr(), cs, off, B, H // 2, W // 2, C_, st)
        _lib.call("pff_avgpool2_bwd", c.data_ptr(), cs, off, acc.data_ptr(), cs, off, B, H, W, C_, 1, st)
        g, y = rows(fine, off), rows(fine2, off)
        d = torch.zeros(C_, device="cuda")
        _lib.call("pff_relu_bias_bwd", g.data_ptr(), cs, off, y.data_ptr(), cs, off, d.data_ptr(), B * H * W, C_, st)
        db.append(d.double())
        res.append([t[:, off:off + C_].contiguous().view(torch.int16) for t in (dn, up, ub, acc, g)])
    for a, b in zip(*res):
        assert torch.equal(a, b)
    # f32 sums of n values in two orders: each within n 2^-24 of the sum of magnitudes
    mag = (fine.double().abs() * (fine2.double() > 0)).sum(0)
    assert ((db[0] - db[1]).abs() <= 2 * B * H * W * 2.0 ** -24 * mag + 1e-30).all()


def test_pow53_is_the_double_power_over_its_whole_range(cuda):
    """Every float of [2^-70, 2^70], where the short form is taken, and an octave beyond: 1.2 G values."""
    from pyfastflow_b200 import _lib

    bad = C.c_longlong(-1)
    _lib.call("pff_pow53_selfcheck", 0x1C000000, 0x63000000, C.byref(bad))
    assert bad.value == 0
