"""Kernels and dispatch rules at the sizes where they can go wrong: edges of tiles, remainders,
the smallest sizes, views that a cluster of blocks shares, against the FP64 oracle, the general
path of the same library or an FP64 torch restatement.  Bar of the projectors and regularisers:
1e-5 relative, as in the parity tests (32-bit sums)."""
import ctypes as C

import numpy as np
import pytest

from tests import geometries as G
from oracle import oracle as O
from tigre_b200.utilities.geometry import cone_geometry

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _geo(shape, det, pix, dso=1000.0, dsd=1536.0, offsets=False, mode="cone"):
    g = cone_geometry(shape, [float(s) for s in shape], det, (pix, pix), DSO=dso, DSD=dsd)
    g.mode = mode
    if offsets:
        g.offOrigin = np.array((1.5, -2.0, 3.25))
        g.offDetector = np.array((2.4, -1.6))
        g.COR = 0.7
    return g


def _plan(geo, ang):
    from tigre_b200 import _native as N
    return N.Plan(N.checked_geometry(geo, ang), 0)


def _close(got, ref, tol=TOL):
    mx, l2 = G.rel_err(got, ref)
    assert mx <= tol and l2 <= tol, (mx, l2)


# ------------------------------------------------------- backprojection: views over a cluster --
@pytest.mark.parametrize("shape,views", [
    ((64, 64, 64), 33),      # 16 tiles: 8 blocks share 33 views (4 or 5 each)
    ((65, 17, 33), 16),      # ragged tiles in every axis, 4 blocks of 4 views
    ((5, 3, 2), 9),          # one tile, odd views over 2 blocks
    ((20, 40, 36), 7),       # too few views to share
])
@pytest.mark.parametrize("kind", ["FDK", "matched"])
def test_backprojection_with_shared_views(shape, views, kind):
    import torch
    from tigre_b200 import _native as N, projectors as P
    geo = _geo(shape, (40, 52), 2.0)
    ang = G.angles(views)
    proj = np.random.default_rng(views).random((views, 40, 52), dtype=np.float32)
    plan = _plan(geo, ang)
    d = torch.from_numpy(proj).cuda()
    ref = O.atb(proj, geo, ang, kind)
    got = P.atb(d, plan, kind)
    _close(got.cpu().numpy(), ref)
    assert torch.equal(got, P.atb(d, plan, kind))            # a fixed order of the sums
    half = P.atb(d, plan, kind, out_dtype=torch.bfloat16).float().cpu().numpy()
    _close(half, ref, 2.0 ** -8)                              # one rounding to BF16
    N.check(N.lib().tigre_atb_ex(plan.handle, C.c_void_p(d.data_ptr()), N.F32, C.c_void_p(got.data_ptr()), N.F32,
                                 P.BACKPROJECTORS[kind], 0, views, 1, None), "tigre_atb_ex")
    _close(got.cpu().numpy(), 2.0 * ref)                      # accumulation
    assert plan.status() == 0


# ------------------------------------------------------------------- Siddon: z-fast working copy --
@pytest.mark.parametrize("shape,det", [
    ((64, 64, 64), (33, 40)),      # four elements per access on both sides
    ((63, 5, 62), (20, 21)),       # rows of the volume no multiple of four
    ((7, 9, 68), (256, 12)),       # rows in fours, runs of the copy shorter than a tile
    ((130, 66, 132), (513, 9)),    # one past a tile in every axis
])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("shift", [0, 1])   # the volume starts on an odd element of a larger buffer
def test_siddon_over_the_zfast_copy(shape, det, dtype, shift):
    import torch
    from tigre_b200 import projectors as P
    geo = _geo(shape, det, 160.0 / max(det), offsets=True)
    ang = G.angles(5)
    dt = getattr(torch, dtype)
    n = int(np.prod(shape))
    flat = torch.from_numpy(np.random.default_rng(n).random(n + shift, dtype=np.float32)).cuda().to(dt)
    vol = flat[shift:].view(shape)
    ref = O.ax(vol.float().cpu().numpy(), geo, ang, "Siddon")
    _close(P.ax(vol, _plan(geo, ang), "Siddon", out_dtype=torch.float32).cpu().numpy(), ref)


# Cells are listed 32 at a time: lists that end in a full one, start a new one for a single cell, and
# crossings of both axes at one point (45 degrees); 8, 4 and 2 rows per thread with remainders.
@pytest.mark.parametrize("xy", [(1, 1), (16, 16), (17, 16), (33, 31), (32, 33), (96, 97)])
@pytest.mark.parametrize("nv", [3, 65, 200, 257])
@pytest.mark.parametrize("mode", ["cone", "parallel"])
def test_siddon_cell_lists(xy, nv, mode):
    import torch
    from tigre_b200 import projectors as P
    shape = (24, xy[1], xy[0])
    geo = _geo(shape, (nv, 14), 40.0 / nv, offsets=True, mode=mode)
    geo.dDetector = np.array((40.0 / nv, 1.7 * max(xy) / 14))
    geo.sDetector = geo.nDetector * geo.dDetector
    ang = np.array([0.0, 0.25, 0.5, 0.31, 0.75, 1.25, 1.5, 1.9]) * np.pi
    vol = np.random.default_rng(nv).random(shape, dtype=np.float32)
    got = P.ax(torch.from_numpy(vol).cuda(), _plan(geo, ang.astype(np.float32)), "Siddon")
    _close(got.cpu().numpy(), O.ax(vol, geo, ang.astype(np.float32), "Siddon"))


@pytest.mark.parametrize("nv", [31, 64, 70, 128, 129, 250, 257])
@pytest.mark.parametrize("mode", ["cone", "parallel"])
def test_siddon_rows_per_thread(nv, mode):
    """A thread takes 2, 4 or 8 rows by the scan's size; a ray's arithmetic does not depend on it.  Columns and
    views that fill the chip against one view at a time (two rows a thread), bit for bit."""
    import torch
    from tigre_b200 import projectors as P
    shape = (24, 17, 19)
    geo = _geo(shape, (nv, 60), 40.0 / nv, offsets=True, mode=mode)
    geo.dDetector = np.array((40.0 / nv, 0.6))
    geo.sDetector = geo.nDetector * geo.dDetector
    plan = _plan(geo, G.angles(75))
    vol = torch.from_numpy(np.random.default_rng(nv).random(shape, dtype=np.float32)).cuda()
    got = P.ax(vol, plan, "Siddon")
    one = torch.cat([P.ax(vol, plan, "Siddon", angle_range=(i, i + 1)) for i in range(75)])
    assert torch.equal(got, one) and float(got.max()) > 1.0


@pytest.mark.parametrize("nz,vox", [(20, 0.1), (20, 0.3), (24, 1.1)])
@pytest.mark.parametrize("nv", [5, 65, 257])
def test_siddon_row_beside_a_slice_plane(nz, vox, nv):
    """An odd number of rows over an even number of slices: the central row runs in the middle plane, and
    with a voxel size that FP32 does not hold that plane comes out less than half an FP32 step of z above
    the row.  Such a row counts as on the plane and reads the slice above, in its whole length."""
    import torch
    from tigre_b200 import projectors as P
    side = np.float64(np.float32(nz * vox)) / 2 / np.float64(np.float32(vox))
    assert 0 < nz / 2 - side < 0.5 * float(np.spacing(np.float32(nz / 2 + 3.99)))   # four slices of pad and more
    shape = (nz, 18, 22)
    geo = cone_geometry(shape, [n * vox for n in shape], (nv, 9), (vox * 40.0 / nv, vox * 4.0), DSO=1000.0 * vox,
                        DSD=1536.0 * vox)
    ang = G.angles(7)
    vol = np.random.default_rng(nz).random(shape, dtype=np.float32)
    got = P.ax(torch.from_numpy(vol).cuda(), _plan(geo, ang), "Siddon").cpu().numpy()
    ref = O.ax(vol, geo, ang, "Siddon")
    vol[nz // 2 - 1] = vol[nz // 2]      # the row's value, whichever of the two slices the oracle takes
    ref[:, nv // 2] = O.ax(vol, geo, ang, "Siddon")[:, nv // 2]
    _close(got, ref)


@pytest.mark.parametrize("nv", [24, 100, 256])
def test_siddon_copy_beyond_one_window(nv):
    """A working copy larger than 4 GB, so that its addresses differ in their high words, against the
    stepped column kernel; the steepest rows leave the volume through its faces."""
    import torch
    from tigre_b200 import _native as N, projectors as P
    shape = (48, 4500, 4400)
    geo = _geo(shape, (nv, 6), 100.0 / nv, dso=20000.0, dsd=30000.0, offsets=True)
    geo.dDetector = np.array((100.0 / nv, 1000.0))
    geo.sDetector = geo.nDetector * geo.dDetector
    ang = np.linspace(0.0, 2.0, 4, dtype=np.float32)
    vol = torch.rand(shape, device="cuda", generator=torch.Generator("cuda").manual_seed(nv))
    got = P.ax(vol, _plan(geo, ang), "Siddon")
    with N.option(N.OPT_SIDDON_KERNEL, 1):
        ref = P.ax(vol, _plan(geo, ang), "Siddon")
    assert float(ref.max()) > 100.0
    _close(got.cpu().numpy(), ref.cpu().numpy(), 2 * TOL)


# --------------------------------------------------------- backprojection: tilted frames --
@pytest.mark.parametrize("shape", [(64, 16, 16), (65, 17, 18), (3, 30, 5), (130, 20, 33)])
@pytest.mark.parametrize("kind", ["FDK", "matched"])
def test_tilted_backprojection(shape, kind):
    import torch
    from tigre_b200 import projectors as P
    geo = _geo(shape, (150, 60), 1.6)
    geo.rotDetector = np.array((0.03, -0.02, 0.05))
    ang = G.angles(11, tilt=True)
    proj = np.random.default_rng(1).random((11, 150, 60), dtype=np.float32)
    got = P.atb(torch.from_numpy(proj).cuda(), _plan(geo, ang), kind).cpu().numpy()
    _close(got, O.atb(proj, geo, ang, kind))


# ---------------------------------------------------------------------------- regularisers --
TV_SHAPES = [(1, 1, 1), (1, 24, 30), (2, 25, 31), (5, 23, 61), (40, 49, 29), (3, 1, 95), (67, 7, 2)]


@pytest.mark.parametrize("shape", TV_SHAPES)
def test_tv_descents(shape):
    import torch
    from tigre_b200 import projectors as P
    rng = np.random.default_rng(5)
    img = rng.random(shape, dtype=np.float32)
    prior = rng.random(shape, dtype=np.float32)

    def dev(a):
        return torch.from_numpy(a.copy()).cuda()
    _close(P.tv_pocs_(dev(img), 0.01, 3).cpu().numpy(), O.pocs_tv(img, 0.01, 3))
    _close(P.tv_aw_pocs_(dev(img), 0.01, 3, 0.3).cpu().numpy(), O.aw_pocs_tv(img, 0.01, 3, 0.3))
    if int(np.prod(shape)) > 1:      # PICCS divides by |g|, which is 0 for a single voxel
        _close(P.tv_piccs_(dev(img), dev(prior), 0.01, 0.4, 3).cpu().numpy(), O.piccs_tv(img, prior, 0.01, 0.4, 3))


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 16, 30), (1, 17, 31), (9, 15, 62), (35, 33, 28)])
@pytest.mark.parametrize("iters", [0, 1, 2, 7])
def test_denoise_in_one_pass_per_iteration(shape, iters):
    import torch
    from tigre_b200 import _native as N
    img = np.random.default_rng(6).random(shape, dtype=np.float32)
    nz, ny, nx = shape
    L = N.lib()
    spacing = (C.c_float * 3)(1.0, 0.5, 2.0)
    out = {}
    for name, floats in (("two", L.tigre_tv_denoise_work_floats(nx, ny, nz)),
                         ("one", L.tigre_tv_denoise_fused_floats(nx, ny, nz))):
        src = torch.from_numpy(img).cuda()
        work = torch.full((floats,), float("nan"), device="cuda")       # no state is read before it is written
        for alias in (False, True):
            dst = src if alias else torch.empty_like(src)
            N.check(L.tigre_tv_denoise_ex(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), nx, ny, nz, 5.0,
                                          C.cast(spacing, C.c_void_p), iters, C.c_void_p(work.data_ptr()), floats,
                                          None), "tigre_tv_denoise_ex")
            torch.cuda.synchronize()
            out[name, alias] = dst.cpu().numpy()
    for key in out:
        _close(out[key], out["two", False], 1e-6)                       # the same recurrences
    rc = L.tigre_tv_denoise_ex(C.c_void_p(src.data_ptr()), C.c_void_p(src.data_ptr()), nx, ny, nz, 5.0, None, 1,
                               C.c_void_p(work.data_ptr()), 1, None)
    assert rc == 4 and "work space" in N.last_error()


@pytest.mark.parametrize("room", [6.0, 8.5, 9.0])
def test_denoise_where_memory_is_short(room, monkeypatch):
    """The result and five floats per voxel of work space always did; the larger work space is taken only
    where the result fits beside it."""
    import torch
    from tigre_b200.utilities.im_3d_denoise import tv_denoise_device
    x = torch.from_numpy(np.random.default_rng(8).random((20, 24, 30), dtype=np.float32)).cuda()
    want = tv_denoise_device(x, 5, 5.0)
    left = [room * 22 / 20 * x.numel()]      # of the padded volume
    alloc = {k: getattr(torch, k) for k in ("empty", "empty_like")}

    def short(name):
        def f(a, *args, **kw):
            n = a.numel() if torch.is_tensor(a) else int(np.prod(a))
            if n > left[0]:
                raise torch.OutOfMemoryError("CUDA out of memory (the test's)")
            left[0] -= n
            return alloc[name](a, *args, **kw)
        return f
    for k in alloc:
        monkeypatch.setattr(torch, k, short(k))
    got = tv_denoise_device(x, 5, 5.0)
    monkeypatch.undo()
    _close(got.cpu().numpy(), want.cpu().numpy(), 1e-6)


# ---------------------------------------------------------------------------- convolutions --
def _conv64(x, w, cout):
    import torch
    k = w.double().view(cout, 3, 3, 3, -1).permute(0, 4, 1, 2, 3)
    return torch.nn.functional.conv3d(x.double().permute(3, 0, 1, 2)[None], k, padding=1)


@pytest.mark.parametrize("D,H,W,cin,cout", [
    (1, 1, 1, 16, 16), (4, 4, 16, 16, 32), (5, 17, 9, 32, 16), (3, 15, 33, 48, 64), (9, 20, 8, 16, 48),
])
def test_convolution_and_its_gradients(D, H, W, cin, cout):
    """Bars: BF16 rounding of the outputs (2^-9 each, 2.5e-3 in all), FP32 sums for the weight and
    bias gradients (1e-5) given the kernel's own ReLU mask."""
    import torch
    from tigre_b200 import _native as N, warmstart
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn((D, H, W, cin), device="cuda", generator=g).bfloat16().requires_grad_(True)
    w = (0.1 * torch.randn((cout, 27 * cin), device="cuda", generator=g)).bfloat16().float().requires_grad_(True)
    b = torch.randn(cout, device="cuda", generator=g).requires_grad_(True)
    dy = torch.randn((D, H, W, cout), device="cuda", generator=g).bfloat16()
    y = warmstart.conv3d(x, w, b, True)
    y.backward(dy)
    x5 = x.detach().double().requires_grad_(True)
    w5 = w.detach().double().requires_grad_(True)
    ref = _conv64(x5, w5, cout) + b.detach().double()[None, :, None, None, None]
    masked = dy.double() * (y.detach() > 0)
    ref.backward(masked.permute(3, 0, 1, 2)[None])

    def rel(a, r):
        return float((a.double() - r).norm() / r.norm().clamp_min(1e-30))
    assert rel(y.detach(), ref.detach().relu()[0].permute(1, 2, 3, 0)) < 2.5e-3
    assert rel(x.grad, x5.grad) < 2.5e-3
    assert rel(w.grad, w5.grad) < 1e-5
    assert rel(b.grad, masked.sum(dim=(0, 1, 2))) < 1e-5
    assert N.lib().tigre_conv3d_status(1) == 0


@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("n,c", [(1, 8), (1000, 24), (70, 2048), (4097, 16)])
def test_relu_and_bias_gradient(n, c, relu):
    """NaN, infinities and -0 go through as dy * (y > 0) gives them."""
    import torch
    from tigre_b200 import _native as N
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    dy = torch.randn((n, c), device="cuda", generator=g).bfloat16()
    y = torch.randn((n, c), device="cuda", generator=g).bfloat16()
    if n > 1:
        dy[1, 0], dy[0, 1], y[0, 1] = float("nan"), float("inf"), -1.0
    out, db = torch.empty_like(dy), torch.empty(c, device="cuda")
    work = torch.empty(N.lib().tigre_conv3d_relu_grad_work(n, c), device="cuda")
    N.check(N.lib().tigre_conv3d_relu_grad(C.c_void_p(dy.data_ptr()), C.c_void_p(y.data_ptr()),
                                           C.c_void_p(out.data_ptr()), C.c_void_p(db.data_ptr()), n, c, relu,
                                           C.c_void_p(work.data_ptr()), None),
            "tigre_conv3d_relu_grad")
    ref = dy.float() * (y > 0) if relu else dy.float()
    if relu:
        assert torch.equal(out.view(torch.int16)[~ref.isnan()], ref.bfloat16().view(torch.int16)[~ref.isnan()])
        assert bool(out[ref.isnan()].isnan().all())
    want = ref.double().sum(0)
    fine = want.isfinite()
    assert torch.equal(fine, db.isfinite())
    # FP32 sums of n terms in a tree: relative to the sum of magnitudes
    size = ref.abs().double().sum(0)
    assert bool(((db.double() - want).abs() <= 1e-5 * size)[fine].all())


@pytest.mark.parametrize("c", [8, 16, 32])
@pytest.mark.parametrize("D,H,W", [(1, 1, 1), (2, 8, 62), (17, 9, 65), (33, 7, 126)])
def test_first_and_last_convolution(c, D, H, W):
    """Bar: one BF16 rounding of the convolution's value (2^-8 of its size)."""
    import torch
    from tigre_b200 import _native as N
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    L, p = N.lib(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    vol = torch.randn((D, H, W), device="cuda", generator=g)
    w = torch.randn((c, 27), device="cuda", generator=g).bfloat16()
    b = torch.randn(c, device="cuda", generator=g)
    y = torch.empty((D, H, W, c), dtype=torch.bfloat16, device="cuda")
    N.check(L.tigre_unet_conv_in(p(vol), p(w), p(b), p(y), D, H, W, c, 0, None), "conv_in")
    ref = (_conv64(vol.bfloat16()[..., None], w, c) + b.double()[None, :, None, None, None])[0].permute(1, 2, 3, 0)
    assert float((y.double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max())
    x = torch.randn((D, H, W, c), device="cuda", generator=g).bfloat16()
    wo = torch.randn((1, 27 * c), device="cuda", generator=g).bfloat16()
    out = torch.empty_like(vol)
    N.check(L.tigre_unet_conv_out(p(x), c, p(wo), 0.25, p(vol), p(out), D, H, W, None), "conv_out")
    ref = _conv64(x, wo, 1)[0, 0] + 0.25
    assert float((out.double() - vol.double() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max()) + 1e-6


@pytest.mark.parametrize("c", [8, 16, 32])
@pytest.mark.parametrize("D,H,W", [(1, 1, 1), (8, 8, 8), (17, 9, 65), (33, 40, 31), (70, 17, 33)])
def test_first_and_last_convolution_order(c, D, H, W):
    """Every sum starts at the bias and takes taps, then channels, in order by FP32 fused multiply-adds: the
    same bits.  (BF16 products are exact in FP64 and so is their sum with an FP32 value 2^29 times larger
    or smaller at most, so that one rounding to FP32 is the fused operation.)"""
    import torch
    from tigre_b200 import _native as N
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    L, p = N.lib(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    shifts = [(t // 9, t // 3 % 3, t % 3) for t in range(27)]

    def taps(v):     # (27, D, H, W, ...) of the zero-padded volume, in FP64
        q = torch.zeros((D + 2, H + 2, W + 2) + v.shape[3:], dtype=torch.float64, device="cuda")
        q[1:-1, 1:-1, 1:-1] = v.double()
        return [q[z:z + D, y:y + H, x:x + W] for z, y, x in shifts]
    vol = torch.randn((D, H, W), device="cuda", generator=g)
    w = torch.randn((c, 27), device="cuda", generator=g).bfloat16()
    b = torch.randn(c, device="cuda", generator=g)
    y = torch.empty((D, H, W, c), dtype=torch.bfloat16, device="cuda")
    N.check(L.tigre_unet_conv_in(p(vol), p(w), p(b), p(y), D, H, W, c, 1, None), "conv_in")
    acc = b.expand(D, H, W, c)
    for t, v in enumerate(taps(vol.bfloat16())):
        acc = (acc.double() + v[..., None] * w[:, t].double()).float()
    assert torch.equal(y, acc.relu().bfloat16())
    x = torch.randn((D, H, W, c), device="cuda", generator=g).bfloat16()
    wo = torch.randn((27, c), device="cuda", generator=g).bfloat16()
    out = torch.empty_like(vol)
    N.check(L.tigre_unet_conv_out(p(x), c, p(wo), 0.25, p(vol), p(out), D, H, W, None), "conv_out")
    acc = torch.full_like(vol, 0.25)
    for t, v in enumerate(taps(x)):
        for k in range(c):
            acc = (acc.double() + v[..., k] * wo[t, k].double()).float()
    assert torch.equal(out, vol + acc.bfloat16().float())


@pytest.mark.parametrize("D,H,W", [(4, 16, 8), (5, 17, 9)])
@pytest.mark.parametrize("cin,cout", [(32, 32), (16, 16)])
def test_convolution_into_any_address(D, H, W, cin, cout):
    """Outputs that do not start on 16 bytes take the kernels with single-element stores: the same
    values but for the order of FP32 sums (27 cin terms) and, in BF16, the step to the neighbouring value that
    it can cause (eight significant bits: 2^-7 of the value at most)."""
    import torch
    from tigre_b200 import _native as N
    g = torch.Generator(device="cuda")
    g.manual_seed(8)
    L, p = N.lib(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    x = torch.randn((D, H, W, cin), device="cuda", generator=g).bfloat16()
    w = torch.randn((cout, 27 * cin), device="cuda", generator=g).bfloat16()
    dy = torch.randn((D, H, W, cout), device="cuda", generator=g).bfloat16()
    col = torch.empty(2 * 27 * D * H * W * max(cin, cout), dtype=torch.bfloat16, device="cuda")
    n, ref, got = D * H * W, {}, {}
    for out, shift in ((ref, 0), (got, 1)):
        yb = torch.empty(n * cout + shift, dtype=torch.bfloat16, device="cuda")[shift:]
        yf = torch.empty(n * cout + shift, device="cuda")[shift:]
        dx = torch.empty(n * cin + shift, device="cuda")[shift:]
        for y, args in ((yb, (p(yb), None)), (yf, (None, p(yf)))):
            N.check(L.tigre_conv3d_fwd(p(x), p(w), None, *args, D, H, W, cin, cout, 0, p(col), None), "fwd")
        N.check(L.tigre_conv3d_bwd_data(p(dy), p(w), p(dx), D, H, W, cin, cout, p(col), None), "bwd_data")
        out.update(yb=yb.double(), yf=yf.double(), dx=dx.double())
    size = 27 * max(cin, cout) * float(x.abs().max() * w.abs().max() + dy.abs().max() * w.abs().max())
    for k, v in ref.items():
        bar = 2.0 ** -23 * size + (2.0 ** -7 * v.abs() if k == "yb" else 0.0)
        assert bool(((got[k] - v).abs() <= bar).all()), k
    half = torch.empty(n * cout + 1, dtype=torch.bfloat16, device="cuda")[1:]
    rc = L.tigre_conv3d_fwd_pair(p(x), cin // 2, p(x), cin // 2, p(w), None, p(half), D, H, W, cout, 0, p(col), None)
    assert rc != 0


@pytest.mark.parametrize("at", [(-1, -1, -1), (-1, 2, 3), (0, -1, 5), (1, 3, -1), (2, 2, 15)])
@pytest.mark.parametrize("D,H,W", [(5, 6, 17), (4, 5, 31), (7, 4, 16)])
def test_weight_gradient_beside_an_infinite_activation(D, H, W, at):
    """An infinite voxel shows in the taps that use it and in no other."""
    import torch
    from tigre_b200 import _native as N
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    cin, cout = 32, 48
    x = torch.randn((D, H, W, cin), device="cuda", generator=g).bfloat16()
    dy = torch.randn((D, H, W, cout), device="cuda", generator=g).bfloat16()
    dy[dy == 0] = 1.0
    x[at][3] = float("inf")
    col = torch.empty(27 * D * H * W * cin, dtype=torch.bfloat16, device="cuda")
    dw = torch.zeros((cout, 27, cin), device="cuda")
    N.check(N.lib().tigre_conv3d_bwd_weight(C.c_void_p(x.data_ptr()), C.c_void_p(dy.data_ptr()), C.c_void_p(dw.data_ptr()),
                                            D, H, W, cin, cout, C.c_void_p(col.data_ptr()), None), "bwd_weight")
    ref = torch.empty((cout, 27, cin), dtype=torch.float64, device="cuda")
    for t in range(27):      # overlapping parts only: no padding to multiply
        a, b = [], []
        for n, o in ((D, t // 9 - 1), (H, t // 3 % 3 - 1), (W, t % 3 - 1)):
            a.append(slice(max(0, -o), n - max(0, o)))
            b.append(slice(max(0, o), n + min(0, o)))
        ref[:, t] = dy[tuple(a)].double().reshape(-1, cout).T @ x[tuple(b)].double().reshape(-1, cin)
    fine = ref.isfinite()
    assert not bool(fine.all()) and torch.equal(fine, dw.isfinite())
    assert torch.equal(ref[~fine], dw[~fine].double())
    assert float((dw[fine].double() - ref[fine]).norm() / ref[fine].norm()) < 1e-5


@pytest.mark.parametrize("threads", [False, True])
def test_convolutions_that_overlap(threads):
    """Training steps of four layers at once, each on a stream of its own from one thread or on one stream from a
    thread each, give what they give one after the other."""
    import threading
    import torch
    from tigre_b200 import warmstart
    g = torch.Generator(device="cuda")
    g.manual_seed(10)
    layers = []
    for cin, cout in ((16, 32), (32, 32), (64, 16), (48, 64)):
        x = torch.randn((20, 17, 24, cin), device="cuda", generator=g).bfloat16()
        w = torch.randn((cout, 27 * cin), device="cuda", generator=g) * 0.05
        dy = torch.randn((20, 17, 24, cout), device="cuda", generator=g).bfloat16()
        layers.append((x, w, torch.zeros(cout, device="cuda"), dy))

    def step(layer):
        x, w, b = (t.detach().requires_grad_(True) for t in layer[:3])
        y = warmstart.conv3d(x, w, b, True)
        y.backward(layer[3])
        return [y.detach(), x.grad, w.grad, b.grad]
    want = [step(layer) for layer in layers]
    torch.cuda.synchronize()
    got = [[] for _ in layers]
    if threads:
        def work(i):
            got[i].extend(step(layers[i]) for _ in range(15))
        ts = [threading.Thread(target=work, args=(i,)) for i in range(len(layers))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    else:
        streams = [torch.cuda.Stream() for _ in layers]
        for _ in range(15):
            for i, st in enumerate(streams):
                with torch.cuda.stream(st):
                    got[i].append(step(layers[i]))
    torch.cuda.synchronize()
    for i, outs in enumerate(got):
        assert len(outs) == 15
        for o in outs:
            assert all(torch.equal(a, b) for a, b in zip(o, want[i])), i


@pytest.mark.parametrize("D,H,W,cin,cout", [(5, 6, 7, 16, 32), (4, 16, 8, 32, 32), (1, 1, 1, 16, 16), (6, 5, 4, 24, 40),
                                            (3, 4, 5, 5, 6), (9, 8, 7, 48, 64)])
def test_convolution_scratch_of_the_stated_size(D, H, W, cin, cout):
    """The calls stay inside the elements that the size queries state, and those inside the im2col matrix."""
    import torch
    from tigre_b200 import _native as N
    L, p = N.lib(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    x = torch.ones((D, H, W, cin), device="cuda").bfloat16()
    w = torch.ones((cout, 27 * cin), device="cuda").bfloat16()
    dy = torch.ones((D, H, W, cout), device="cuda").bfloat16()
    y, dw = torch.empty_like(dy), torch.zeros((cout, 27 * cin), device="cuda")
    full = int(L.tigre_conv3d_col_elems(D, H, W, cin))
    fwd, bwd = (int(f(D, H, W, cin, cout)) for f in (L.tigre_conv3d_fwd_work, L.tigre_conv3d_bwd_weight_work))
    assert 0 < fwd <= full and 0 < bwd <= full
    for n, call in ((fwd, lambda c: L.tigre_conv3d_fwd(p(x), p(w), None, p(y), None, D, H, W, cin, cout, 0, c, None)),
                    (bwd, lambda c: L.tigre_conv3d_bwd_weight(p(x), p(dy), p(dw), D, H, W, cin, cout, c, None))):
        col = torch.full((full + 64,), 7.0, device="cuda").bfloat16()      # what lies behind stays
        N.check(call(p(col)), "conv3d")
        assert bool((col[n:] == 7.0).all())


def test_convolution_under_saved_tensor_hooks():
    """A hook that gives the saved tensors back at odd addresses: the same gradients up to the order of FP32
    sums in the kernels that take such inputs."""
    import torch
    from tigre_b200 import warmstart
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    leaves = [torch.randn((6, 7, 9, 16), device="cuda", generator=g).bfloat16(),
              torch.randn((32, 27 * 16), device="cuda", generator=g) * 0.05, torch.randn(32, device="cuda", generator=g)]
    dy = torch.randn((6, 7, 9, 32), device="cuda", generator=g).bfloat16()

    def shifted(t):
        return torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)

    def step():
        x, w, b = (t.detach().requires_grad_(True) for t in leaves)
        warmstart.conv3d(x, w, b, True).backward(dy)
        return x.grad.double(), w.grad.double(), b.grad.double()
    want = step()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, shifted):
        got = step()
    for a, b, bar in zip(got, want, (2.5e-3, 1e-5, 1e-5)):     # bars of test_convolution_and_its_gradients
        assert float((a - b).norm() / b.norm()) < bar


@pytest.mark.parametrize("D,H,W", [(4, 16, 8), (6, 18, 10), (9, 7, 23), (8, 4, 4)])
@pytest.mark.parametrize("ca,cb,cout", [(16, 48, 32), (64, 16, 16), (32, 32, 64)])
def test_convolution_of_a_pair(D, H, W, ca, cb, cout):
    """Two inputs where they are: the bits of the convolution of their concatenation."""
    import torch
    from tigre_b200 import _native as N
    g = torch.Generator(device="cuda")
    g.manual_seed(12)
    L, p = N.lib(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    xa = torch.randn((D, H, W, ca), device="cuda", generator=g).bfloat16()
    xb = torch.randn((D, H, W, cb), device="cuda", generator=g).bfloat16()
    w = (0.1 * torch.randn((cout, 27 * (ca + cb)), device="cuda", generator=g)).bfloat16()
    b = torch.randn(cout, device="cuda", generator=g)
    x = torch.cat([xa, xb], dim=-1)
    y, ref = (torch.empty((D, H, W, cout), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    n = 27 * (ca + cb) * cout
    col = torch.full((n + 64,), 7.0, device="cuda").bfloat16()
    assert L.tigre_conv3d_fwd_pair_ok(D, H, W, ca, cb, cout) == 1
    N.check(L.tigre_conv3d_fwd_pair(p(xa), ca, p(xb), cb, p(w), p(b), p(y), D, H, W, cout, 1, p(col), None), "pair")
    assert bool((col[n:] == 7.0).all())
    N.check(L.tigre_conv3d_fwd(p(x), p(w), p(b), p(ref), None, D, H, W, ca + cb, cout, 1, p(col), None), "fwd")
    assert torch.equal(y, ref) and bool(ref.any())


@pytest.mark.parametrize("d,h,w,c", [(1, 1, 1, 8), (3, 5, 7, 24), (16, 17, 9, 16)])
def test_upsampling(d, h, w, c):
    import torch
    from tigre_b200 import _native as N
    x = torch.arange(d * h * w * c, device="cuda").remainder(251).view(d, h, w, c).bfloat16()
    out = torch.empty((2 * d, 2 * h, 2 * w, c), dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().tigre_unet_up2(C.c_void_p(x.data_ptr()), C.c_void_p(out.data_ptr()), 2 * d, 2 * h, 2 * w, c, None), "up2")
    assert torch.equal(out, x.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2))


@pytest.mark.parametrize("D,H,W,halo", [(200, 1, 200, 0), (200, 2, 200, 0), (40, 3, 300, 0), (200, 5, 200, 1), (50, 50, 50, 1),
                                        (96, 1, 1, 1), (5, 16, 8, 1), (200, 200, 1, 0)])
def test_convolution_of_thin_volumes(D, H, W, halo):
    """Volumes much thinner than a tile keep the kernels that gather voxels; both give the FP64 convolution.
    Bars of test_convolution_and_its_gradients."""
    import torch
    from tigre_b200 import _native as N
    g = torch.Generator(device="cuda")
    g.manual_seed(13)
    L, p = N.lib(), lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    cin, cout = 32, 48
    assert L.tigre_conv3d_fwd_pair_ok(D, H, W, 16, 16, cout) == halo
    x = torch.randn((D, H, W, cin), device="cuda", generator=g).bfloat16()
    w = (0.1 * torch.randn((cout, 27 * cin), device="cuda", generator=g)).bfloat16()
    dy = torch.randn((D, H, W, cout), device="cuda", generator=g).bfloat16()
    y, dx = torch.empty_like(dy), torch.empty((D, H, W, cin), device="cuda")
    col = torch.empty(2 * 27 * D * H * W * cin, dtype=torch.bfloat16, device="cuda")
    N.check(L.tigre_conv3d_fwd(p(x), p(w), None, p(y), None, D, H, W, cin, cout, 0, p(col), None), "fwd")
    N.check(L.tigre_conv3d_bwd_data(p(dy), p(w), p(dx), D, H, W, cin, cout, p(col), None), "bwd_data")
    ref = _conv64(x, w, cout)[0].permute(1, 2, 3, 0)
    assert float((y.double() - ref).norm() / ref.norm()) < 2.5e-3
    wt = w.view(cout, 27, cin).flip(1).permute(2, 1, 0).reshape(cin, 27 * cout)
    ref = _conv64(dy, wt, cin)[0].permute(1, 2, 3, 0)
    assert float((dx.double() - ref).norm() / ref.norm()) < 1e-5

