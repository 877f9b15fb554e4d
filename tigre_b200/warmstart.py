"""Learned CGLS warm start: a small 3D U-Net that maps a sparse-view FDK reconstruction to
CGLS's initial image.

Everything runs on the device: the convolutions are this library's BF16 tensor-core kernels
(tigre_conv3d_fwd / _bwd_data / _bwd_weight, FP32 accumulation) wrapped as a
torch.autograd.Function; pooling, upsampling, concatenation and the optimiser are PyTorch
plumbing.  Training pairs are generated by the library itself: seeded random-ellipsoid
phantoms, Siddon projections with Poisson noise (CTnoise) and the 100-iteration CGLS
reconstruction as target, or noiseless projections with the phantom as target; FDK is the
input.  Two losses: the squared error to the target, and (whole volumes) a data term, the
relative residual |b - A x|^2 / |b|^2 either of the network's output or of the k-th CGLS
iterate started from it (unroll = k: the CGLS recurrences run inside the graph, through the
projector pair's autograd Functions).  The second trains the start for what CGLS does with it:
a start with a small residual can still need as many iterations, if its error lies where CGLS
converges slowly.  Plain CGLS (zero or FDK initial image) is the fallback and the comparison.

    python -m tigre_b200.warmstart --train 96 --steps 800 --eval 8 --out result.json
    python -m tigre_b200.warmstart --size 256 --crop 0 --load w.npz --finetune --physics 1e4 \
        --unroll 4 --img-weight 0.1 --clean-frac 0.5 --steps 1000 --lr 1e-4 --save w2.npz

Architecture (4 levels, 16 base channels): two 3x3x3 conv + ReLU per level with channels
16/32/64/128, 2x2x2 average pooling down, nearest-neighbour upsampling and concatenation of
the skip connection up, a final linear 3x3x3 conv to one channel added to the input.  Volumes
are channels-last (D, H, W, C); sizes must be multiples of 8.
"""
from __future__ import annotations

import ctypes as C
import json
import math
import os
import time

import numpy as np

from . import _native as N

SCALE = 50.0   # attenuation (~0.02 / mm) to O(1) network inputs


def _torch():
    import torch
    return torch


def _stream(t):
    from .projectors import _stream as s
    return s(t)


def _col(work, sizes, *inputs):
    """Elements of scratch of a convolution call: work(*sizes) where its inputs start on 16 bytes, else the im2col
    matrix.  Every call allocates its own from its stream's allocator: calls on other streams or from other
    threads cannot meet in it."""
    if any(t.data_ptr() % 16 for t in inputs):
        work, sizes = N.lib().tigre_conv3d_col_elems, sizes[:4]
    return work(*sizes)


def conv3d(x, w, b, relu):
    """y = relu?(conv3d(x, w) + b): x (D, H, W, Cin) BF16 CUDA, w (Cout, 27*Cin) FP32 master
    weights (cast to BF16 for the kernel), b (Cout,) FP32.  Returns BF16 (D, H, W, Cout)."""
    return _ConvFn.apply(x, w, b, bool(relu))


def _conv_fn():
    T = _torch()

    class ConvFn(T.autograd.Function):
        @staticmethod
        def forward(ctx, x, w, b, relu):
            D, H, W, Cin = x.shape
            Cout = w.shape[0]
            x = x.contiguous()
            wb = w.to(T.bfloat16).contiguous()
            y = T.empty((D, H, W, Cout), dtype=T.bfloat16, device=x.device)
            col = T.empty(_col(N.lib().tigre_conv3d_fwd_work, (D, H, W, Cin, Cout), x, wb), dtype=T.bfloat16,
                          device=x.device)
            N.check(N.lib().tigre_conv3d_fwd(C.c_void_p(x.data_ptr()), C.c_void_p(wb.data_ptr()),
                                             C.c_void_p(b.data_ptr()), C.c_void_p(y.data_ptr()), None, D, H, W, Cin,
                                             Cout, 1 if relu else 0, C.c_void_p(col.data_ptr()), _stream(x)),
                    "tigre_conv3d_fwd")
            ctx.save_for_backward(x, wb, y)
            ctx.relu = relu
            return y

        @staticmethod
        def backward(ctx, dy):
            x, wb, y = ctx.saved_tensors
            D, H, W, Cin = x.shape
            Cout = wb.shape[0]
            L = N.lib()
            # the fused pass reads 16 bytes at a time; y may be what a saved-tensor hook made of it
            fused = dy.dtype == T.bfloat16 and Cout % 8 == 0 and Cout <= 2048 and dy.contiguous().data_ptr() % 16 == 0 \
                and not (ctx.relu and (y.dtype != T.bfloat16 or not y.is_contiguous() or y.data_ptr() % 16))
            # one scratch for the three steps, which run one after the other (the other inputs of the two
            # convolutions are allocated here, on 16 bytes)
            col = T.empty(max(_col(L.tigre_conv3d_bwd_weight_work, (D, H, W, Cin, Cout), x),
                              L.tigre_conv3d_fwd_work(D, H, W, Cout, Cin) if Cout % 8 == 0 else 0,
                              2 * L.tigre_conv3d_relu_grad_work(D * H * W, Cout) if fused else 0),
                          dtype=T.bfloat16, device=x.device)
            if fused:
                # ReLU mask and bias sums in one pass
                dy = dy.contiguous()
                gb = T.empty_like(dy) if ctx.relu else dy
                db = T.empty(Cout, dtype=T.float32, device=x.device)
                N.check(L.tigre_conv3d_relu_grad(C.c_void_p(dy.data_ptr()), C.c_void_p(y.data_ptr()),
                                                 C.c_void_p(gb.data_ptr()), C.c_void_p(db.data_ptr()), D * H * W,
                                                 Cout, 1 if ctx.relu else 0, C.c_void_p(col.data_ptr()),
                                                 _stream(x)), "tigre_conv3d_relu_grad")
            else:
                g = dy.float()
                if ctx.relu:
                    g = g * (y > 0)
                db = g.sum(dim=(0, 1, 2))
                gb = g.to(T.bfloat16).contiguous()
            if Cout % 8 == 0:
                dx = T.empty((D, H, W, Cin), dtype=T.bfloat16, device=x.device)
                # the data gradient is the forward convolution of dy with the tap-flipped,
                # channel-transposed weights: wt[c][t*Cout + co] = w[co][(26 - t)*Cin + c]
                wt = wb.view(Cout, 27, Cin).flip(1).permute(2, 1, 0).reshape(Cin, 27 * Cout).contiguous()
                N.check(L.tigre_conv3d_fwd(C.c_void_p(gb.data_ptr()), C.c_void_p(wt.data_ptr()), None,
                                           C.c_void_p(dx.data_ptr()), None, D, H, W, Cout, Cin, 0,
                                           C.c_void_p(col.data_ptr()), _stream(x)), "tigre_conv3d_fwd")
            else:
                dx = T.empty((D, H, W, Cin), dtype=T.float32, device=x.device)
                dcol = T.empty(int(L.tigre_conv3d_col_elems(D, H, W, Cin)), dtype=T.float32, device=x.device)
                N.check(L.tigre_conv3d_bwd_data(C.c_void_p(gb.data_ptr()), C.c_void_p(wb.data_ptr()),
                                                C.c_void_p(dx.data_ptr()), D, H, W, Cin, Cout,
                                                C.c_void_p(dcol.data_ptr()), _stream(x)), "tigre_conv3d_bwd_data")
            dw = T.zeros((Cout, 27 * Cin), dtype=T.float32, device=x.device)
            N.check(L.tigre_conv3d_bwd_weight(C.c_void_p(x.data_ptr()), C.c_void_p(gb.data_ptr()),
                                              C.c_void_p(dw.data_ptr()), D, H, W, Cin, Cout,
                                              C.c_void_p(col.data_ptr()), _stream(x)), "tigre_conv3d_bwd_weight")
            return dx.to(T.bfloat16), dw, db, None

    return ConvFn


class _Lazy:
    def __init__(self, make):
        self._make = make
        self._obj = None

    def __getattr__(self, name):
        if self._obj is None:
            self._obj = self._make()
        return getattr(self._obj, name)


_ConvFn = _Lazy(_conv_fn)


def _make_unet_class():
    T = _torch()
    nn = T.nn

    class Conv(nn.Module):
        def __init__(self, cin, cout, relu=True):
            super().__init__()
            fan_in = 27 * cin
            self.w = nn.Parameter(T.randn(cout, fan_in) * math.sqrt(2.0 / fan_in))
            self.b = nn.Parameter(T.zeros(cout))
            self.relu = relu

        def forward(self, x):
            return conv3d(x, self.w, self.b, self.relu)

    def pool(x):
        D, H, W, Cc = x.shape
        return x.float().view(D // 2, 2, H // 2, 2, W // 2, 2, Cc).mean(dim=(1, 3, 5)).to(T.bfloat16)

    def up(x):
        return x.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)

    class UNet3D(nn.Module):
        def __init__(self, base=16, levels=4):
            super().__init__()
            ch = [base * (2 ** i) for i in range(levels)]
            self.enc = nn.ModuleList()
            cin = 1
            for c in ch:
                self.enc.append(nn.ModuleList([Conv(cin, c), Conv(c, c)]))
                cin = c
            self.dec = nn.ModuleList()
            for i in range(levels - 2, -1, -1):
                self.dec.append(nn.ModuleList([Conv(ch[i + 1] + ch[i], ch[i]), Conv(ch[i], ch[i])]))
            self.head = Conv(ch[0], 1, relu=False)

        def forward(self, vol):
            """vol: (D, H, W) FP32 in network units; returns (D, H, W) FP32.  Without autograd
            (inference) the fused pass `infer` runs instead, with the same arithmetic."""
            if not (T.is_grad_enabled() and any(p.requires_grad for p in self.parameters())) and self.fused_ok(vol):
                return self.infer(vol)
            x = vol.to(T.bfloat16).unsqueeze(-1).contiguous()
            skips = []
            for i, (c1, c2) in enumerate(self.enc):
                x = c2(c1(x))
                if i < len(self.enc) - 1:
                    skips.append(x)
                    x = pool(x)
            for (c1, c2), s in zip(self.dec, reversed(skips)):
                x = T.cat([up(x), s], dim=-1).contiguous()
                x = c2(c1(x))
            return vol + self.head(x).float().squeeze(-1)

        def fused_ok(self, vol):
            levels = len(self.enc)
            return (vol.is_cuda and vol.dim() == 3 and all(d % (2 ** (levels - 1)) == 0 for d in vol.shape)
                    and self.enc[0][0].w.shape[0] in (8, 16, 32) and all(c.w.shape[0] % 8 == 0 for c, _ in self.enc))

        @T.no_grad()
        def infer(self, vol):
            """The forward pass with this library's kernels: the first and last convolutions (one
            input / one output channel) in FP32, the others on the tensor cores, pooling and
            upsampling in one pass each; the decoder's convolutions read the upsampled level and the
            skip connection where they are, or a concatenated copy where they cannot."""
            L = N.lib()
            st = _stream(vol)
            vol = vol.float().contiguous()
            D, H, W = vol.shape
            p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

            def conv(x, layer):
                d, h, w, cin = x.shape
                cout = layer.w.shape[0]
                y = T.empty((d, h, w, cout), dtype=T.bfloat16, device=x.device)
                wb = self._wbf(layer)
                col = T.empty(_col(L.tigre_conv3d_fwd_work, (d, h, w, cin, cout), x, wb), dtype=T.bfloat16, device=x.device)
                N.check(L.tigre_conv3d_fwd(p(x), p(wb), p(layer.b), p(y), None, d, h, w, cin, cout,
                                           1 if layer.relu else 0, p(col), st), "tigre_conv3d_fwd")
                return y

            c1 = self.enc[0][0]
            x = T.empty((D, H, W, c1.w.shape[0]), dtype=T.bfloat16, device=vol.device)
            N.check(L.tigre_unet_conv_in(p(vol), p(self._wbf(c1)), p(c1.b), p(x), D, H, W, c1.w.shape[0],
                                         1 if c1.relu else 0, st), "tigre_unet_conv_in")
            x = conv(x, self.enc[0][1])
            skips = []
            for i in range(1, len(self.enc)):
                skips.append(x)
                d, h, w, c = x.shape
                pooled = T.empty((d // 2, h // 2, w // 2, c), dtype=T.bfloat16, device=x.device)
                N.check(L.tigre_unet_pool2(p(x), p(pooled), d, h, w, c, st), "tigre_unet_pool2")
                x = conv(conv(pooled, self.enc[i][0]), self.enc[i][1])
            for (ca, cb), s in zip(self.dec, reversed(skips)):
                d, h, w, cs = s.shape
                cx, co = x.shape[-1], ca.w.shape[0]
                if L.tigre_conv3d_fwd_pair_ok(d, h, w, cx, cs, co):
                    # the convolution reads the upsampled level and the skip connection where they are
                    up = T.empty((d, h, w, cx), dtype=T.bfloat16, device=x.device)
                    N.check(L.tigre_unet_up2(p(x), p(up), d, h, w, cx, st), "tigre_unet_up2")
                    y = T.empty((d, h, w, co), dtype=T.bfloat16, device=x.device)
                    col = T.empty(27 * (cx + cs) * co, dtype=T.bfloat16, device=x.device)
                    N.check(L.tigre_conv3d_fwd_pair(p(up), cx, p(s), cs, p(self._wbf(ca)), p(ca.b), p(y), d, h, w, co,
                                                    1 if ca.relu else 0, p(col), st), "tigre_conv3d_fwd_pair")
                    x = conv(y, cb)
                    continue
                cat = T.empty((d, h, w, x.shape[-1] + cs), dtype=T.bfloat16, device=x.device)
                N.check(L.tigre_unet_up_concat(p(x), x.shape[-1], p(s), cs, p(cat), d, h, w, st),
                        "tigre_unet_up_concat")
                x = conv(conv(cat, ca), cb)
            out = T.empty_like(vol)
            head = self.head
            N.check(L.tigre_unet_conv_out(p(x), x.shape[-1], p(self._wbf(head)), float(head.b.detach()[0].item()),
                                          p(vol), p(out), D, H, W, st), "tigre_unet_conv_out")
            return out

        def _wbf(self, layer):
            """BF16 copy of a layer's weights, kept while the FP32 master weights are unchanged."""
            key = (layer.w.data_ptr(), layer.w._version)
            cache = getattr(layer, "_wbf_cache", None)
            if cache is None or cache[0] != key:
                cache = (key, layer.w.detach().to(T.bfloat16).contiguous())
                layer._wbf_cache = cache
            return cache[1]

        def flops(self, shape):
            """Multiply-add FLOPs (x2) of one forward pass on a (D, H, W) volume."""
            n = int(np.prod(shape))
            total, lev = 0, 0
            for c1, c2 in self.enc:
                v = n // (8 ** lev)
                for c in (c1, c2):
                    total += 2 * c.w.shape[0] * c.w.shape[1] * v
                lev += 1
            for i, (c1, c2) in enumerate(self.dec):
                v = n // (8 ** (len(self.enc) - 2 - i))
                for c in (c1, c2):
                    total += 2 * c.w.shape[0] * c.w.shape[1] * v
            total += 2 * self.head.w.shape[0] * self.head.w.shape[1] * n
            return total

    return UNet3D


UNet3D = _Lazy(_make_unet_class)


def unet(base=16, levels=4, device="cuda", seed=0):
    T = _torch()
    T.manual_seed(seed)
    cls = _make_unet_class()
    return cls(base, levels).to(device)


# --------------------------------------------------------------------------- data --

def problem_geometry(n=128):
    """The warm-start problem, C5 scaled to n^3: 256 mm cube, detector 2n x 2n at 0.8*256/n mm,
    DSO 1000, DSD 1536, 90 views over 2 pi."""
    from .utilities.geometry import cone_geometry
    det = 2 * n
    return cone_geometry((n, n, n), (256.0, 256.0, 256.0), (det, det), (0.8 * 256 / n, 0.8 * 256 / n),
                         DSO=1000.0, DSD=1536.0)


def angles(nviews=90):
    a = np.zeros((nviews, 3), dtype=np.float32)
    a[:, 0] = np.linspace(0, 2 * np.pi, nviews, endpoint=False)
    return a


PRETRAINED_C5 = os.path.join(os.path.dirname(os.path.abspath(__file__)), "data", "unet_c5_256cube_90views.npz")


def save_weights(model, path):
    """The network's parameters in an .npz file: convolution weights as the BF16 values the
    kernels use (their 16 bits, key "<name>.bf16"), biases in FP32."""
    out = {}
    for k, v in model.state_dict().items():
        a = v.detach().float().cpu().numpy()
        if k.endswith(".w"):
            b = a.view(np.uint32).astype(np.uint64)
            out[k + ".bf16"] = ((b + 0x7FFF + ((b >> 16) & 1)) >> 16).astype(np.uint16)   # nearest even
        else:
            out[k] = a
    np.savez_compressed(path, **out)


def load_weights(model, path):
    state = np.load(path)
    T = _torch()
    params = {}
    for k in state.files:
        if k.endswith(".bf16"):
            params[k[:-5]] = T.from_numpy((state[k].astype(np.uint32) << 16).view(np.float32))
        else:
            params[k] = T.from_numpy(state[k])
    model.load_state_dict(params)
    return model


def pretrained_c5(device="cuda"):
    """The U-Net trained on the warm-start configuration (256^3 @ 1 mm, 512^2 @ 0.8 mm, 90 views),
    or None.  Training, all with this library's kernels on seeded phantoms: 2000 Adam steps on
    64^3 crops against 100-iteration CGLS targets of 96 noisy (I0 = 5e4) cases; then on whole
    volumes of 48 noisy and 48 noiseless cases, 600 steps adding the start's own relative
    residual (weight 100), then 400 + 800 + 1000 steps on the relative residual after 4 / 5 / 4
    unrolled CGLS iterations (weight 1e4, image term 0.1, learning rate 2e-4 / 1.5e-4 / 1e-4)."""
    if not os.path.exists(PRETRAINED_C5):
        return None
    return load_weights(unet(device="cpu"), PRETRAINED_C5).to(device)


def make_pair(seed, n=128, nviews=90, I0=5e4, cgls_iters=100, clean=False):
    """(projections, FDK input, target, phantom) on the device, for phantom `seed`: noisy
    projections with the 100-iteration CGLS reconstruction as target, or with clean=True the
    noiseless projections with the phantom itself as target."""
    T = _torch()
    from .algorithms._common import Problem
    from .algorithms.krylov import cgls_device
    from .algorithms.single_pass import fdk_device
    from .utilities import CTnoise
    from .utilities.phantom import random_ellipsoids
    from . import projectors as P
    geo, ang = problem_geometry(n), angles(nviews)
    img = random_ellipsoids((n, n, n), seed=seed, device="cuda")
    plan = N.get_plan(N.checked_geometry(geo, ang), img.device.index)
    proj = P.ax(img, plan, "Siddon")
    if clean:
        prob = Problem(proj, geo, ang)
        return proj, fdk_device(prob), img, img
    noisy = CTnoise.add(proj, Poisson=float(I0), Gaussian=np.array([0.0, 0.5]), seed=1000003 + seed)
    noisy = T.nan_to_num(noisy, nan=0.0, posinf=0.0, neginf=0.0).contiguous()
    prob = Problem(noisy, geo, ang)
    fdk = fdk_device(prob)
    target, _, _ = cgls_device(prob, cgls_iters)
    return noisy, fdk, target, img


def train(model, n_train=96, steps=400, n=128, crop=64, lr=1e-3, seed=0, log=None, physics=0.0, clean_frac=0.0,
          img_weight=1.0, unroll=0):
    """Adam (cosine learning-rate decay to 1 %) on img_weight x the squared error to the target
    (the 100-iteration CGLS reconstruction of noisy data, or the phantom for the clean_frac
    share of noiseless pairs); with physics > 0 (whole volumes only) the loss adds
    physics * |A x - b|^2 / |b|^2, the relative data residual that the warm-started CGLS then
    reduces, through the projector's autograd Function (backward = matched Atb).  With
    unroll = k > 0 the data term is instead the relative residual after k CGLS iterations from
    the network's output (the iteration differentiated through its projections and scalars):
    the start is trained for what CGLS does with it, not for its own residual."""
    T = _torch()
    t0 = time.perf_counter()
    data = []
    plan = None
    n_clean = int(round(clean_frac * n_train))
    for s in range(n_train):
        b, fdk, target, _ = make_pair(10000 + s, n=n, clean=s < n_clean)
        data.append((fdk * SCALE, target * SCALE, b if physics > 0 else None))
    if physics > 0:
        if crop and crop < n:
            raise ValueError("the data term needs whole volumes (crop=0)")
        from .autograd import AtbFunction, AxFunction
        plan = N.get_plan(N.checked_geometry(problem_geometry(n), angles()), data[0][0].device.index)
    t_data = time.perf_counter() - t0
    opt = T.optim.Adam(model.parameters(), lr=lr)
    sched = T.optim.lr_scheduler.CosineAnnealingLR(opt, T_max=max(steps, 1), eta_min=lr * 0.01)
    rng = np.random.default_rng(seed)
    losses = []
    t1 = time.perf_counter()
    for it in range(steps):
        x, y, b = data[rng.integers(len(data))]
        if crop and crop < n:
            o = rng.integers(0, n - crop + 1, size=3) // 8 * 8
            x = x[o[0]:o[0] + crop, o[1]:o[1] + crop, o[2]:o[2] + crop]
            y = y[o[0]:o[0] + crop, o[1]:o[1] + crop, o[2]:o[2] + crop]
        pred = model(x.contiguous())
        loss = img_weight * T.mean((pred - y) ** 2)
        if physics > 0:
            r = b - AxFunction.apply((pred / SCALE).contiguous(), plan, "Siddon")
            if unroll > 0:
                # CGLS (krylov.py's recurrences) from the prediction, k steps, residual only
                s = AtbFunction.apply(r.contiguous(), plan, "matched")
                p, gamma = s, (s * s).sum()
                for i in range(unroll):
                    q = AxFunction.apply(p.contiguous(), plan, "Siddon")
                    r = r - (gamma / (q * q).sum()) * q
                    if i + 1 < unroll:
                        s = AtbFunction.apply(r.contiguous(), plan, "matched")
                        g_new = (s * s).sum()
                        p, gamma = s + (g_new / gamma) * p, g_new
            loss = loss + physics * (r * r).sum() / (b * b).sum()
        opt.zero_grad()
        loss.backward()
        opt.step()
        sched.step()
        losses.append(float(loss.item()))
        if log and (it % 50 == 0 or it == steps - 1):
            log("step %d loss %.6f" % (it, losses[-1]))
    T.cuda.synchronize()
    return {"n_train": n_train, "steps": steps, "crop": crop, "data_seconds": t_data,
            "train_seconds": time.perf_counter() - t1, "loss_first": losses[0], "loss_last": float(np.mean(losses[-20:])),
            "physics": physics, "clean_frac": clean_frac, "img_weight": img_weight, "lr": lr, "unroll": unroll}


def cgls_to_residual(prob, x0, target_rel, max_iter=300):
    """CGLS from x0 until |b - A x| / |b| <= target_rel; returns (iterations, seconds, reached)."""
    T = _torch()
    from .algorithms.krylov import cgls_device
    T.cuda.synchronize()
    t = time.perf_counter()
    _, res, _ = cgls_device(prob, max_iter, x0=x0, tol=target_rel)
    T.cuda.synchronize()
    bnorm = float(T.linalg.vector_norm(prob.b.double()).item())
    rel = res / bnorm
    hit = np.nonzero(rel <= target_rel)[0]
    return (int(hit[0]) + 1 if hit.size else len(rel)), time.perf_counter() - t, bool(hit.size)


def evaluate(model, n_eval=8, n=128, nviews=90, log=None, noiseless_target=None):
    """Time to a residual target for plain CGLS (zero / FDK start) and the warm start (U-Net
    inference included).  With noisy data the relative residual stalls at the noise level, far
    above 1e-3, so the target is that of 100 plain zero-start iterations, plus 0.1 %.  With
    noiseless_target set, the data are the noiseless projections and the target that value."""
    T = _torch()
    from .algorithms._common import Problem
    from .algorithms.krylov import cgls_device
    from .algorithms.single_pass import fdk_device
    from . import projectors as P
    rows = []
    for s in range(n_eval):
        noisy, _, _, img = make_pair(20000 + s, n=n, nviews=nviews, cgls_iters=1)
        if noiseless_target is not None:
            plan = N.get_plan(N.checked_geometry(problem_geometry(n), angles(nviews)), img.device.index)
            noisy = P.ax(img, plan, "Siddon")
        prob = Problem(noisy, problem_geometry(n), angles(nviews))
        bnorm = float(T.linalg.vector_norm(prob.b.double()).item())
        if noiseless_target is not None:
            target = float(noiseless_target)
        else:
            _, res100, _ = cgls_device(prob, 100)
            target = float(res100[-1] / bnorm) * 1.001
        it0, t0, ok0 = cgls_to_residual(prob, None, target)
        T.cuda.synchronize()
        tf = time.perf_counter()
        f = fdk_device(prob).clamp_(min=0)
        T.cuda.synchronize()
        t_fdk = time.perf_counter() - tf
        itf, tff, okf = cgls_to_residual(prob, f, target)
        T.cuda.synchronize()
        tw = time.perf_counter()
        with T.no_grad():
            x0 = (model(fdk_device(prob) * SCALE) / SCALE).contiguous()
        T.cuda.synchronize()
        t_inf = time.perf_counter() - tw
        itw, tww, okw = cgls_to_residual(prob, x0, target)
        plan = N.get_plan(N.checked_geometry(problem_geometry(n), angles(nviews)), img.device.index)
        rel0 = lambda x: float(T.linalg.vector_norm((P.ax(x, plan, "Siddon") - prob.b).double()).item()) / bnorm  # noqa: E731
        row = {"seed": 20000 + s, "target_rel_residual": target, "plain_zero": {"iters": it0, "s": t0, "reached": ok0},
               "plain_fdk": {"iters": itf, "s": t_fdk + tff, "reached": okf, "start_rel_residual": rel0(f)},
               "warm": {"iters": itw, "s": t_inf + tww, "inference_s": t_inf, "reached": okw,
                        "start_rel_residual": rel0(x0)}}
        rows.append(row)
        if log:
            log(json.dumps(row))
    med = lambda k: float(np.median([r[k]["s"] for r in rows]))  # noqa: E731
    return {"cases": rows, "median_s": {k: med(k) for k in ("plain_zero", "plain_fdk", "warm")},
            "warm_over_plain_zero": med("warm") / med("plain_zero"),
            "warm_over_plain_fdk": med("warm") / med("plain_fdk")}


def main(argv=None):
    import argparse
    ap = argparse.ArgumentParser(description=__doc__.split("\n")[0])
    ap.add_argument("--train", type=int, default=96)
    ap.add_argument("--steps", type=int, default=800)
    ap.add_argument("--eval", type=int, default=8)
    ap.add_argument("--size", type=int, default=128)
    ap.add_argument("--crop", type=int, default=0)
    ap.add_argument("--physics", type=float, default=0.0)
    ap.add_argument("--lr", type=float, default=1e-3)
    ap.add_argument("--out", default=None)
    ap.add_argument("--save", default=None, help="write the trained weights to this .npz")
    ap.add_argument("--load", default=None, help="skip training: load weights from this .npz")
    ap.add_argument("--finetune", action="store_true", help="with --load: train on from the loaded weights")
    ap.add_argument("--clean-frac", type=float, default=0.0, help="share of noiseless training pairs")
    ap.add_argument("--img-weight", type=float, default=1.0)
    ap.add_argument("--unroll", type=int, default=0, help="data term after this many CGLS iterations")
    ap.add_argument("--noiseless-target", type=float, default=5e-3)
    args = ap.parse_args(argv)
    model = unet()
    tr = {}
    if args.load:
        load_weights(model, args.load)
        tr["loaded"] = args.load
    if not args.load or args.finetune:
        tr.update(train(model, args.train, args.steps, args.size, args.crop, lr=args.lr, log=print, physics=args.physics,
                        clean_frac=args.clean_frac, img_weight=args.img_weight, unroll=args.unroll))
        if args.save:
            save_weights(model, args.save)
    ev = evaluate(model, args.eval, args.size, log=print)
    ev0 = evaluate(model, args.eval, args.size, log=print, noiseless_target=args.noiseless_target)
    res = {"train": tr, "eval_noisy": ev, "eval_noiseless": ev0,
           "unet_gflop_per_inference": model.flops((args.size,) * 3) / 1e9}
    print(json.dumps(res))
    if args.out:
        json.dump(res, open(args.out, "w"), indent=1)


if __name__ == "__main__":
    main()
