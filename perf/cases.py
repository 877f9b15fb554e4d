"""The work that users of this framework have it do, as measurable cases.

Every case goes through a public entry point with what a user's program keeps in hand (plans,
operator modules, a network with its weights):

  ax, atb, pair   projectors.ax / projectors.atb on device tensors with a kept plan
  autograd        autograd.create_pytorch_operator and autograd.tv, forward and backward
  cgls            algorithms.cgls on device projections
  tv, denoise     projectors.tv_pocs_ and utilities.im_3d_denoise.im3ddenoise
  unet, conv      the warm-start network's inference and one convolution layer's training step

Inputs are made from the seed alone and without this framework's projectors: ellipsoid phantoms
(attenuations up to 0.02 / mm), their analytic line integrals with measurement noise, and
Gaussian activations and weights.  exact() restates every operation in FP64 torch.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from tigre_b200 import _native as N
from tigre_b200 import algorithms, autograd, projectors, warmstart
from tigre_b200.utilities.geometry import cone_geometry
from tigre_b200.utilities.im_3d_denoise import im3ddenoise

DEV = "cuda"
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
DSO, DSD = 1000.0, 1536.0
LAMBDA_TV = 1e-3      # weight of the TV term of the autograd case


# ------------------------------------------------------------------------------------ cases --
def _scan(name, kind, shape, vox, det, pix, views, **more):
    c = {"name": name, "kind": kind, "nz": shape[0], "ny": shape[1], "nx": shape[2], "vox": vox,
         "nv": det[0], "nu": det[1], "pix": pix, "views": views, "first": 0, "count": views,
         "proj": "Siddon", "back": "matched", "dtype": "f32", "tilt": False, "offsets": False,
         "batch": 1, "iters": 0}
    c.update(more)
    return c


def listed():
    return [
        # the small plain-method configuration: one projection and one backprojection of it, where
        # launches and occupancy count
        _scan("ax_siddon_64", "ax", (64, 64, 64), 1.0, (128, 128), 0.8, 100),
        _scan("atb_matched_64", "atb", (64, 64, 64), 1.0, (128, 128), 0.8, 100),
        # the benchmark's step: the projector pair over a full scan of the largest volume
        _scan("pair_512", "pair", (512, 512, 512), 0.5, (768, 1024), 0.4, 720),
        # one OS-SART subset of the reduced-storage configuration: 36 of the 720 views, FDK weights
        _scan("subset_512_bf16", "pair", (512, 512, 512), 0.5, (768, 1024), 0.4, 720, first=216, count=36,
              back="FDK", dtype="bf16"),
        # the fixed-step projector over the mid-size scan
        _scan("ax_interp_256", "ax", (256, 256, 256), 1.0, (512, 512), 0.8, 360, proj="interpolated"),
        # a general trajectory (tilted detector, non-axial Euler angles, offsets) at odd sizes
        _scan("pair_tilted_ragged", "pair", (181, 203, 190), 1.0, (233, 251), 1.3, 77, tilt=True, offsets=True),
        # the differentiable operator: |Ax - b|^2 + TV over a batch, forward and backward
        _scan("autograd_128", "autograd", (128, 128, 128), 1.0, (256, 256), 0.8, 180, batch=8),
        # a whole reconstruction: CGLS iterations on the sparse-view scan
        _scan("cgls_256", "cgls", (256, 256, 256), 1.0, (512, 512), 0.8, 90, iters=10),
        # the regularisers of ASD-POCS (20 descent steps per sweep) and of FISTA / SART-TV (defaults)
        {"name": "tv_pocs_ragged", "kind": "tv", "nz": 301, "ny": 333, "nx": 317, "iters": 20},
        {"name": "denoise_256", "kind": "denoise", "nz": 256, "ny": 256, "nx": 256, "iters": 50},
        # the learned warm start: one inference, and one layer's forward and backward in training
        {"name": "unet_infer_256", "kind": "unet", "nz": 256, "ny": 256, "nx": 256},
        {"name": "conv_train_64", "kind": "conv", "nz": 64, "ny": 64, "nx": 64, "cin": 32, "cout": 32},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ax", "ax", "atb", "atb", "pair", "autograd", "cgls", "tv", "denoise", "unet", "conv"])
    if kind in ("tv", "denoise"):
        return {"kind": kind, "nz": _log(rng, 24, 360), "ny": _log(rng, 24, 360), "nx": _log(rng, 24, 360),
                "iters": rng.randint(4, 30)}
    if kind == "unet":
        return {"kind": kind, "nz": 8 * _log(rng, 4, 28), "ny": 8 * _log(rng, 4, 28), "nx": 8 * _log(rng, 4, 28)}
    if kind == "conv":
        return {"kind": kind, "nz": _log(rng, 12, 96), "ny": _log(rng, 12, 96), "nx": _log(rng, 12, 96),
                "cin": rng.choice([16, 32, 48, 64]), "cout": rng.choice([16, 32, 64])}
    heavy = kind in ("autograd", "cgls")
    n = _log(rng, 40, 144 if heavy else 400)
    shape = [max(16, int(n * rng.uniform(0.7, 1.1))) for _ in range(3)]
    vox = round(rng.choice([1.0, 256.0 / n]), 4)
    nu = max(32, int(n * rng.uniform(1.3, 2.1)))
    pix = round(1.62 * vox * max(shape) / nu, 4)
    nv = max(32, int(nu * shape[0] / max(shape) * rng.uniform(0.7, 1.0)))
    views = _log(rng, 24, 180) if heavy else _log(rng, 8, 360)
    count = views if heavy or rng.random() < 0.5 else _log(rng, 1, views)
    tilt = (not heavy) and rng.random() < 0.25
    proj = "Siddon" if heavy or tilt else rng.choice(["Siddon", "Siddon", "interpolated"])
    if proj == "interpolated":
        nu, nv, count = min(nu, 480), min(nv, 480), min(count, 120)
    c = _scan("", kind, shape, vox, (nv, nu), pix, views, first=rng.randint(0, views - count), count=count,
              proj=proj, back="matched" if heavy else rng.choice(["matched", "FDK"]),
              dtype="f32" if heavy else rng.choice(["f32", "f32", "bf16", "f16"]), tilt=tilt,
              offsets=tilt or rng.random() < 0.3, batch=rng.randint(1, 6) if kind == "autograd" else 1,
              iters=rng.randint(3, 12) if kind == "cgls" else 0)
    del c["name"]
    return c


# --------------------------------------------------------------------------------- geometry --
def _geometry(c):
    shape = (c["nz"], c["ny"], c["nx"])
    g = cone_geometry(shape, [s * c["vox"] for s in shape], (c["nv"], c["nu"]), (c["pix"], c["pix"]), DSO=DSO, DSD=DSD)
    if c["offsets"]:
        g.offOrigin = np.array((1.5, -2.0, 3.25)) * c["vox"]
        g.offDetector = np.array((2.4, -1.6)) * c["pix"]
        g.COR = 0.7 * c["vox"]
    a = np.zeros((c["views"], 3), dtype=np.float32)
    a[:, 0] = np.linspace(0.0, 2.0 * np.pi, c["views"], endpoint=False)
    if c["tilt"]:
        g.rotDetector = np.array((0.03, -0.02, 0.05))
        r = np.random.default_rng(3)
        a[:, 1] = r.uniform(-0.3, 0.3, c["views"])
        a[:, 2] = r.uniform(-0.3, 0.3, c["views"])
    return g, a


def _rz(t):
    c, s = math.cos(t), math.sin(t)
    return np.array([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]])


def _ry(t):
    c, s = math.cos(t), math.sin(t)
    return np.array([[c, 0.0, s], [0.0, 1.0, 0.0], [-s, 0.0, c]])


def _rx(t):
    c, s = math.cos(t), math.sin(t)
    return np.array([[1.0, 0.0, 0.0], [0.0, c, -s], [0.0, s, c]])


class _Exact:
    """The scan in FP64, from the float32 values that the framework's geometry holds."""

    def __init__(self, c):
        g, a = _geometry(c)
        f = lambda v: np.asarray(np.asarray(v, dtype=np.float32), dtype=np.float64)  # noqa: E731
        self.n = np.array([c["nx"], c["ny"], c["nz"]])
        self.d, self.s = f(g.dVoxel)[::-1].copy(), f(g.sVoxel)[::-1].copy()          # x, y, z
        self.off = f(g.offOrigin)[::-1].copy()
        self.nu, self.nv = c["nu"], c["nv"]
        self.du, self.dv = float(f(g.dDetector)[1]), float(f(g.dDetector)[0])
        self.su, self.sv = float(f(g.sDetector)[1]), float(f(g.sDetector)[0])
        self.offu, self.offv = float(f(g.offDetector)[1]), float(f(g.offDetector)[0])
        self.cor = float(f(getattr(g, "COR", 0.0)))
        self.dso, self.dsd = float(np.float32(DSO)), float(np.float32(DSD))
        self.acc = float(np.float32(g.accuracy))
        rot = f(g.rotDetector)
        self.rd = _rz(rot[2]) @ _ry(rot[1]) @ _rx(rot[0])
        self.ang = np.asarray(a, dtype=np.float64)

    def rays(self, i):
        """Source and pixel positions of view i, in mm from the volume's centre plus offsets."""
        al, th, ps = self.ang[i]
        re = _rz(al) @ _ry(th) @ _rz(ps)
        shift = -self.off + np.array([-self.cor * math.sin(al), self.cor * math.cos(al), 0.0])
        src = re @ np.array([self.dso, 0.0, 0.0]) + shift
        base = np.array([-(self.dsd - self.dso), self.offu, self.offv])
        u = (torch.arange(self.nu, dtype=torch.float64, device=DEV) - self.nu / 2 + 0.5) * self.du
        v = (torch.arange(self.nv, dtype=torch.float64, device=DEV) - self.nv / 2 + 0.5) * self.dv
        ru, rv, o = re @ self.rd[:, 1], re @ self.rd[:, 2], re @ base + shift
        pix = [float(o[k]) + u[None, :] * float(ru[k]) + v[:, None] * float(rv[k]) for k in range(3)]
        return src, pix

    def siddon(self, vol, views):
        """Line integrals by exact plane crossings, one slab of the ray's dominant axis at a time."""
        nx, ny, nz = (int(v) for v in self.n)
        flat, out = vol.double().reshape(-1), []
        group = max(1, int(4e6 // (self.nu * self.nv)))
        for g0 in range(0, len(views), group):
            s, r = [[], [], []], [[], [], []]
            for i in views[g0:g0 + group]:
                src, pix = self.rays(i)
                for k in range(3):
                    sk = (src[k] + self.s[k] / 2) / self.d[k]
                    rk = (pix[k] + self.s[k] / 2) / self.d[k] - sk
                    s[k].append(torch.full_like(rk, sk))
                    r[k].append(torch.where(rk.abs() < 1e-3, torch.zeros_like(rk), rk))
            s, r = [torch.stack(v).reshape(-1) for v in s], [torch.stack(v).reshape(-1) for v in r]
            am, aM = torch.full_like(s[0], -1e300), torch.full_like(s[0], 1e300)
            for k in range(3):
                inv = 1.0 / r[k]
                a0, a1 = -s[k] * inv, (float(self.n[k]) - s[k]) * inv
                zero = r[k] == 0
                outside = zero & ((s[k] < 0) | (s[k] > float(self.n[k])))
                am = torch.where(zero, am, torch.maximum(am, torch.minimum(a0, a1)))
                aM = torch.where(zero, aM, torch.minimum(aM, torch.maximum(a0, a1)))
                aM = torch.where(outside, torch.full_like(aM, -1e300), aM)
            R = torch.stack(r)
            dom = R.abs().argmax(0)
            o1, o2 = (dom + 1) % 3, (dom + 2) % 3
            S = torch.stack(s)
            pick = lambda t, k: t.gather(0, k[None])[0]  # noqa: E731
            n = torch.tensor([nx, ny, nz], dtype=torch.float64, device=DEV)
            st = torch.tensor([1, nx, nx * ny], dtype=torch.int64, device=DEV)
            sd, rd, s1, r1, s2, r2 = pick(S, dom), pick(R, dom), pick(S, o1), pick(R, o1), pick(S, o2), pick(R, o2)
            n1, n2, t0, t1, t2 = n[o1] - 1, n[o2] - 1, st[dom], st[o1], st[o2]
            invd = 1.0 / rd
            i1, i2 = torch.where(r1 == 0, torch.zeros_like(r1), 1 / r1), torch.where(r2 == 0, torch.zeros_like(r2), 1 / r2)
            live, total = n[dom], torch.zeros_like(s[0])
            for k in range(max(nx, ny, nz)):
                lo, hi = (k - sd) * invd, (k + 1 - sd) * invd
                a, b = torch.maximum(torch.minimum(lo, hi), am), torch.minimum(torch.maximum(lo, hi), aM)
                b = torch.where(k < live, torch.maximum(a, b), a)
                cut = []
                for sk, rk, ik in ((s1, r1, i1), (s2, r2, i2)):   # at most one plane of each other axis in a slab
                    x, y = sk + a * rk, sk + b * rk
                    p = torch.floor(torch.maximum(x, y))
                    cut.append(torch.where(rk == 0, a, torch.minimum(torch.maximum((p - sk) * ik, a), b)))
                m0, m1 = torch.minimum(cut[0], cut[1]), torch.maximum(cut[0], cut[1])
                kk = t0 * torch.clamp(torch.full_like(live, float(k)), max=live - 1).long()
                for e0, e1 in ((a, m0), (m0, m1), (m1, b)):
                    mid = 0.5 * (e0 + e1)
                    j1 = torch.minimum(torch.clamp(torch.floor(s1 + mid * r1), min=0.0), n1).long()
                    j2 = torch.minimum(torch.clamp(torch.floor(s2 + mid * r2), min=0.0), n2).long()
                    total += (e1 - e0) * flat[kk + j1 * t1 + j2 * t2]
            length = torch.sqrt(sum((r[k] * self.d[k]) ** 2 for k in range(3)))
            out.append((total * length).reshape(-1, self.nv, self.nu))
        return torch.cat(out)

    def interpolated(self, vol, views):
        """Fixed-step trilinear samples with border 0 (axial views)."""
        v5 = vol.double()[None, None]
        nx, ny, nz = (int(v) for v in self.n)
        out = []
        for i in views:
            src, pix = self.rays(i)
            s = [(src[k] + self.s[k] / 2) / self.d[k] - 0.5 for k in range(3)]
            d = [(pix[k] + self.s[k] / 2) / self.d[k] - 0.5 - s[k] for k in range(3)]
            steps = torch.ceil(torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2) / self.acc)
            vec = [t / steps for t in d]
            al = self.ang[i, 0]
            mx, my = nx // 2 + abs(self.off[0]) / self.d[0], ny // 2 + abs(self.off[1]) / self.d[1]
            a, b = self.dso / self.d[0], self.dso / self.d[1]
            near = a * b / math.sqrt((a * math.sin(al)) ** 2 + (b * math.cos(al)) ** 2) - math.sqrt(mx * mx + my * my)
            crop = math.floor(max(near, 0.0))
            first = math.floor(crop / self.acc)
            cap = (2.0 * self.dso / min(self.d[0], self.d[1]) + crop) / self.acc
            last = torch.where(steps > cap, torch.full_like(steps, math.ceil(cap)), steps)
            lo, hi = torch.full_like(steps, first), last
            for k in range(3):
                ta, tb = (-1.0 - s[k]) / vec[k], (float(self.n[k]) - s[k]) / vec[k]
                lo = torch.maximum(lo, torch.nan_to_num(torch.floor(torch.minimum(ta, tb)), neginf=-1e9))
                hi = torch.minimum(hi, torch.nan_to_num(torch.ceil(torch.maximum(ta, tb)), posinf=1e9))
            hit = lo <= hi
            total = torch.zeros_like(steps)
            if bool(hit.any()):
                j0, j1 = int(lo[hit].min()), int(hi[hit].max())
                chunk = max(1, int(1.6e7 // steps.numel()))
                for j in range(j0, j1 + 1, chunk):
                    q = torch.arange(j, min(j + chunk, j1 + 1), dtype=torch.float64, device=DEV)[:, None, None]
                    grid = torch.stack([(s[k] + q * vec[k]) * (2.0 / max(int(self.n[k]) - 1, 1)) - 1.0 for k in range(3)], -1)
                    val = F.grid_sample(v5, grid[None], mode="bilinear", padding_mode="zeros", align_corners=True)[0, 0]
                    total += (val * ((q >= first) & (q <= last))).sum(0)
            out.append(total * torch.sqrt(sum((vec[k] * self.d[k]) ** 2 for k in range(3))))
        return torch.stack(out)

    def backproject(self, proj, views, matched):
        """Bilinear samples at the voxels' projections, weighted and summed (border 0)."""
        nx, ny, nz = (int(v) for v in self.n)
        out = torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEV)
        axis = lambda k, n: -(self.s[k] - self.d[k]) / 2 + self.off[k] + torch.arange(n, dtype=torch.float64, device=DEV) * self.d[k]  # noqa: E731,E501
        X, Y, Z = axis(0, nx)[None, None, :], axis(1, ny)[None, :, None], axis(2, nz)[:, None, None]
        away = self.dsd - self.dso
        for i, view in enumerate(views):
            al, th, ps = self.ang[view]
            rt, rdt = _rz(-ps) @ _ry(-th) @ _rz(-al), self.rd.T
            src = rdt @ np.array([self.dsd, -self.offu, -self.offv])
            src[0] -= away
            m = rdt @ rt
            shift = rdt @ np.array([away, -self.offu, -self.offv])
            shift[0] -= away

            def lin(k):
                t = float(m[k, 0]) * X + float(m[k, 1]) * Y + float(shift[k])
                return t + float(m[k, 2]) * Z if abs(m[k, 2]) > 1e-15 else t
            t = (self.dso - self.dsd - src[0]) / (lin(0) - src[0])
            u = (lin(1) - src[1] - self.cor) * t / self.du + src[1] / self.du + self.nu / 2
            v = (lin(2) - src[2]) * t / self.dv + src[2] / self.dv + self.nv / 2
            grid = torch.stack(torch.broadcast_tensors((2 * u - 1) / max(self.nu - 1, 1) - 1, (2 * v - 1) / max(self.nv - 1, 1) - 1), -1)
            p = proj[i].double()[None, None]
            val = F.grid_sample(p, grid.expand(nz, ny, nx, 2).reshape(1, nz * ny, nx, 2), mode="bilinear",
                                padding_mode="zeros", align_corners=True).reshape(nz, ny, nx)
            ca, sa = math.cos(al), math.sin(al)
            if matched:
                day = u * self.du + (self.du - self.su) / 2 + self.offu
                dx, dy = -away * ca - day * sa, day * ca - away * sa
                dz = v * self.dv + (self.dv - self.sv) / 2 + self.offv
                l2 = (self.dso * ca - dx) ** 2 + (self.dso * sa - dy) ** 2 + dz ** 2
                lsq = (self.dso * ca - X) ** 2 + (self.dso * sa - Y) ** 2 + Z ** 2
                out += val * (l2 * torch.sqrt(l2) / (self.dsd * lsq))
            else:
                out += val * (self.dso / (self.dso - (Y + self.cor) * sa - X * ca)) ** 2
        return out * (float(np.prod(self.d)) / (self.du * self.dv)) if matched else out


# ----------------------------------------------------------------------------------- inputs --
def _generator(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _ellipsoids(seed, half):
    r = np.random.default_rng(int(seed))
    half = np.asarray(half)
    return [(r.uniform(-0.6, 0.6, 3) * half, r.uniform(0.1, 0.8, 3) * half, r.uniform(0.002, 0.01)) for _ in range(10)]


def _phantom(c, seed, vox=1.0, noise=0.0):
    """Sum of ten ellipsoids in / mm, clipped to 0.02, with Gaussian noise."""
    n = (c["nx"], c["ny"], c["nz"])
    ax = [(torch.arange(k, dtype=torch.float32, device=DEV) - (k - 1) / 2) * vox for k in n]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    vol = torch.zeros((n[2], n[1], n[0]), dtype=torch.float32, device=DEV)
    for m, r, v in _ellipsoids(seed, [0.5 * k * vox for k in n]):
        q = ((X - m[0]) / r[0]) ** 2 + ((Y - m[1]) / r[1]) ** 2 + ((Z - m[2]) / r[2]) ** 2
        vol += (q <= 1.0) * float(v)
    vol.clamp_(max=0.02)
    if noise:
        vol += noise * torch.randn(vol.shape, generator=_generator(seed, 1), device=DEV)
    return vol


def _projections(c, seed):
    """Analytic line integrals of the ellipsoids, with noise of the size photon counting gives."""
    e = _Exact(c)
    ells = _ellipsoids(seed, e.s / 2)
    out = torch.empty((c["count"], c["nv"], c["nu"]), dtype=torch.float32, device=DEV)
    for j, i in enumerate(range(c["first"], c["first"] + c["count"])):
        src, pix = e.rays(i)
        d = [(pix[k] - float(src[k])).float() for k in range(3)]
        length = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
        row = torch.zeros_like(length)
        for m, r, v in ells:
            p = [float(src[k] - m[k]) / r[k] for k in range(3)]
            q = [d[k] / float(r[k]) for k in range(3)]
            a = q[0] * q[0] + q[1] * q[1] + q[2] * q[2]
            b = p[0] * q[0] + p[1] * q[1] + p[2] * q[2]
            row += float(v) * torch.sqrt(torch.clamp(b * b - a * (p[0] ** 2 + p[1] ** 2 + p[2] ** 2 - 1.0), min=0.0)) / a
        out[j] = 2.0 * row * length
    out += 0.004 * torch.randn(out.shape, generator=_generator(seed, 2), device=DEV)
    return out


def _network(seed):
    net = warmstart.unet(seed=0)
    with torch.no_grad():
        for k, p in enumerate(net.parameters()):
            if p.dim() == 2:     # BF16 values, as stored weights have
                w = torch.randn(p.shape, generator=_generator(seed, 10 + k), device=DEV) * math.sqrt(2.0 / p.shape[1])
                p.copy_(w.bfloat16().float())
            else:
                p.copy_(0.05 * torch.randn(p.shape, generator=_generator(seed, 10 + k), device=DEV))
    return net


def _activations(c, seed):
    return torch.randn((c["nz"], c["ny"], c["nx"], c["cin"]), generator=_generator(seed, 3), device=DEV).relu().bfloat16()


def _layer(c, seed):
    fan = 27 * c["cin"]
    w = torch.randn((c["cout"], fan), generator=_generator(seed, 4), device=DEV) * math.sqrt(2.0 / fan)
    b = 0.05 * torch.randn(c["cout"], generator=_generator(seed, 5), device=DEV)
    dy = torch.randn((c["nz"], c["ny"], c["nx"], c["cout"]), generator=_generator(seed, 6), device=DEV).bfloat16()
    return w.bfloat16().float(), b, dy


def prepare(case, seed):
    c, s = case, {"case": case}
    if c["kind"] in ("ax", "atb", "pair", "autograd", "cgls"):
        s["geo"], s["angles"] = _geometry(c)
        dt = DTYPES[c["dtype"]]
        if c["kind"] in ("ax", "atb", "pair"):
            s["plan"] = N.get_plan(N.checked_geometry(s["geo"], s["angles"]), 0)
            s["range"] = (c["first"], c["first"] + c["count"])
            if c["kind"] != "atb":
                s["vol"] = _phantom(c, seed, c["vox"]).to(dt)
            if c["kind"] != "ax":
                s["proj"] = _projections(c, seed).to(dt)
        elif c["kind"] == "autograd":
            s["A"], _ = autograd.create_pytorch_operator(s["geo"], s["angles"])
            s["x"] = torch.stack([_phantom(c, 100 * seed + j, c["vox"], 5e-4) for j in range(c["batch"])])
            s["b"] = torch.stack([_projections(c, 100 * seed + j) for j in range(c["batch"])])
        else:
            s["proj"] = _projections(c, seed)
    elif c["kind"] in ("tv", "denoise"):
        s["vol"] = _phantom(c, seed, 1.0, 1e-3)
        s["work"] = torch.empty_like(s["vol"])
        s["alpha"] = _alpha(c)
    elif c["kind"] == "unet":
        s["net"] = _network(0)
        s["vol"] = warmstart.SCALE * _phantom(c, seed, 1.0, 1e-3)
    else:
        s["x"] = _activations(c, seed)
        s["w"], s["b"], s["dy"] = _layer(c, 0)[:2] + (_layer(c, seed)[2],)
    return s


def _alpha(c):
    return 4e-5 * math.sqrt(c["nz"] * c["ny"] * c["nx"])


# ------------------------------------------------------------------------------------- runs --
def run(state):
    c, s = state["case"], state
    kind = c["kind"]
    if kind in ("ax", "atb", "pair"):
        out = {}
        if kind != "atb":
            out["proj"] = projectors.ax(s["vol"], s["plan"], c["proj"], angle_range=s["range"])
        if kind != "ax":
            out["vol"] = projectors.atb(s["proj"], s["plan"], c["back"], angle_range=s["range"])
        return out
    if kind == "autograd":
        x = s["x"].detach().requires_grad_(True)
        loss = ((s["A"](x) - s["b"]) ** 2).sum() + LAMBDA_TV * autograd.tv(x)
        loss.backward()
        return {"loss": loss.detach(), "grad": x.grad}
    if kind == "cgls":
        return algorithms.cgls(s["proj"], s["geo"], s["angles"], c["iters"])
    if kind == "tv":
        return projectors.tv_pocs_(s["vol"].clone(), s["alpha"], c["iters"], work=s["work"])
    if kind == "denoise":
        return im3ddenoise(s["vol"], c["iters"], 15.0)
    if kind == "unet":
        with torch.no_grad():
            return s["net"](s["vol"])
    x, w, b = (s[k].detach().requires_grad_(True) for k in ("x", "w", "b"))
    y = warmstart.conv3d(x, w, b, True)
    y.backward(s["dy"])
    return {"y": y.detach(), "dx": x.grad, "dw": w.grad, "db": b.grad}


# ------------------------------------------------------------------------------------ exact --
def _tv_parts(f):
    """Backward differences of f between zero slices in z (zero across the x and y faces)."""
    dz = F.pad(f, (0, 0, 0, 0, 1, 1))
    dz = dz[1:] - dz[:-1]                                   # nz + 1 planes
    dy = F.pad(f[:, 1:] - f[:, :-1], (0, 0, 1, 0))
    dx = F.pad(f[:, :, 1:] - f[:, :, :-1], (1, 0))
    return dz, F.pad(dy, (0, 0, 0, 0, 0, 1)), F.pad(dx, (0, 0, 0, 0, 0, 1))


def _tv_gradient(f):
    dz, dy, dx = _tv_parts(f)
    n = torch.sqrt(dz * dz + dy * dy + dx * dx) + 1e-8
    dz, dy, dx = dz / n, dy / n, dx / n
    g = dz[:-1] + dy[:-1] + dx[:-1] - dz[1:]
    g[:, :-1] -= dy[:-1, 1:]
    g[:, :, :-1] -= dx[:-1, :, 1:]
    return g


def _exact_denoise(img, iters, lam):
    f0 = img.double()
    lo = f0.min()
    f0 = f0 - lo
    hi = f0.max()
    f0 = f0 / hi
    ghost = f0[1:2] if f0.shape[0] > 1 else torch.zeros_like(f0[:1])
    f = torch.cat([ghost, f0, torch.zeros_like(f0[:1])])
    u, p = f.clone(), [torch.zeros_like(f) for _ in range(3)]
    for i in range(iters):
        t2 = 0.3 + 0.02 * i
        t1 = (1 / t2) * (1 / 6 - 5 / (15 + i))
        div = sum(torch.diff(p[k], dim=k, prepend=torch.zeros_like(p[k].narrow(k, 0, 1))) for k in range(3))
        u = u * (1 - t1) + t1 * (f + div / lam)
        q = [p[k] + t2 * torch.diff(u, dim=k, append=u.narrow(k, u.shape[k] - 1, 1)) for k in range(3)]
        n = torch.clamp(torch.sqrt(q[0] ** 2 + q[1] ** 2 + q[2] ** 2), min=1.0)
        p = [t / n for t in q]
    return u[1:-1] * hi + lo


def _conv64(x, w, b, relu):
    """x (C, D, H, W), w (Cout, 27 Cin) tap-major: one shifted matrix product per tap, channels first."""
    cin = x.shape[0]
    w = w.double().reshape(w.shape[0], 27, cin)
    xp = F.pad(x, (1, 1, 1, 1, 1, 1))
    D, H, W = x.shape[1:]
    y = b.double()[:, None, None, None].expand(-1, D, H, W).clone()
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        y += torch.einsum("oc,cdhw->odhw", w[:, t], xp[:, dz:dz + D, dy:dy + H, dx:dx + W])
    return y.relu() if relu else y


def _exact_unet(net, vol):
    act = lambda x, m: _conv64(x, m.w.detach(), m.b.detach(), m.relu)  # noqa: E731
    x, skips = vol.double()[None], []
    for i, (a, b) in enumerate(net.enc):
        x = act(act(x, a), b)
        if i + 1 < len(net.enc):
            skips.append(x)
            x = F.avg_pool3d(x[None], 2)[0]
    for (a, b), s in zip(net.dec, reversed(skips)):
        x = act(act(torch.cat([F.interpolate(x[None], scale_factor=2, mode="nearest")[0], s]), a), b)
    return vol.double() + act(x, net.head)[0]


def exact(case, seed):
    c = case
    rays = c.get("count", 0) * c.get("nu", 0) * c.get("nv", 0)
    voxels = c["nz"] * c["ny"] * c["nx"]
    span = max(c["nz"], c["ny"], c["nx"])
    if c["kind"] in ("ax", "atb", "pair"):
        s, e, out = prepare(c, seed), _Exact(c), {}
        views = list(range(c["first"], c["first"] + c["count"]))
        if c["kind"] != "atb":
            big = rays * span > 5e10
            out["proj"] = None if big else (e.siddon if c["proj"] == "Siddon" else e.interpolated)(s["vol"], views)
        if c["kind"] != "ax":
            big = voxels * len(views) > 2e10
            out["vol"] = None if big else e.backproject(s["proj"], views, c["back"] == "matched")
        return None if all(v is None for v in out.values()) else out
    if c["kind"] == "autograd":
        s, e = prepare(c, seed), _Exact(c)
        views, loss, grads = list(range(c["views"])), 0.0, []
        for x, b in zip(s["x"], s["b"]):
            r = e.siddon(x, views) - b.double()
            dz, dy, dx = _tv_parts(x.double())
            loss += (r * r).sum() + LAMBDA_TV * torch.sqrt(dz * dz + dy * dy + dx * dx).sum()
            grads.append(2 * e.backproject(r, views, True) + LAMBDA_TV * _tv_gradient(x.double()))
        return {"loss": loss, "grad": torch.stack(grads)}
    if c["kind"] == "cgls":
        if rays * span * c["iters"] > 2e10:
            return None
        s, e = prepare(c, seed), _Exact(c)
        views, r = list(range(c["views"])), s["proj"].double()
        p = e.backproject(r, views, True)
        x, g = torch.zeros_like(p), (p * p).sum()
        for _ in range(c["iters"]):
            q = e.siddon(p, views)
            a = g / (q * q).sum()
            x += a * p
            r = r - a * q
            t = e.backproject(r, views, True)
            g, last = (t * t).sum(), g
            p = t + (g / last) * p
        return x
    if c["kind"] == "tv":
        f, alpha = prepare(c, seed)["vol"].double(), _alpha(c)
        for _ in range(c["iters"]):
            g = _tv_gradient(f)
            f = f - alpha * g / torch.sqrt((g * g).sum() + 1e-7)
        return f
    if c["kind"] == "denoise":
        return _exact_denoise(prepare(c, seed)["vol"], c["iters"], 15.0)
    with torch.no_grad():
        s = prepare(c, seed)
        if c["kind"] == "unet":
            return None if voxels > 160 ** 3 else _exact_unet(s["net"], s["vol"])
        x, w = s["x"].double().permute(3, 0, 1, 2), s["w"].double()
        y = _conv64(x, w, s["b"], True)
        dy = torch.where(y > 0, s["dy"].double().permute(3, 0, 1, 2), torch.zeros_like(y))
        wt = w.reshape(c["cout"], 27, c["cin"]).flip(1).permute(2, 1, 0).reshape(c["cin"], -1)
        dx = _conv64(dy, wt, torch.zeros(c["cin"], dtype=torch.float64, device=DEV), False)
        xp = F.pad(x, (1, 1, 1, 1, 1, 1))
        D, H, W = y.shape[1:]
        dw = torch.stack([torch.einsum("odhw,cdhw->oc", dy, xp[:, t // 9:t // 9 + D, t // 3 % 3:t // 3 % 3 + H,
                                                               t % 3:t % 3 + W]) for t in range(27)], 1)
        last = lambda t: t.permute(1, 2, 3, 0).contiguous()  # noqa: E731
        return {"y": last(y), "dx": last(dx), "dw": dw.reshape(c["cout"], -1), "db": dy.sum(dim=(1, 2, 3))}


# ----------------------------------------------------------------------------- work, bounds --
def work(case):
    """Bytes: inputs and outputs once per operator application.  Flops: a ray crosses about one
    voxel of each in-plane axis's mean extent per step (2 per segment), a trilinear sample is 7
    lerps and an add, a voxel update 3 lerps and a weighted add."""
    c = case
    vox = c["nz"] * c["ny"] * c["nx"]
    if c["kind"] in ("tv", "denoise"):
        # each step needs the whole image before it (a global norm) or the dual field (3 values)
        per = (8, 30) if c["kind"] == "tv" else (36, 30)
        return {"bytes": per[0] * vox * c["iters"], "flops": per[1] * vox * c["iters"]}
    if c["kind"] == "unet":
        flops, n = 0, vox
        ch = [16, 32, 64, 128]
        for i, k in enumerate(ch):
            flops += 2 * 27 * k * ((ch[i - 1] if i else 1) + k) * n / 8 ** i
            if i < 3:
                flops += 2 * 27 * k * (ch[i + 1] + k + k) * n / 8 ** i
        return {"bytes": 8 * vox, "flops": flops + 2 * 27 * 16 * n}
    if c["kind"] == "conv":
        return {"bytes": vox * (4 * c["cin"] + 4 * c["cout"]), "flops": 3 * 2 * 27 * c["cin"] * c["cout"] * vox}
    rays, es = c["count"] * c["nu"] * c["nv"], 4 if c["dtype"] == "f32" else 2
    crossed = rays * 0.5 * (c["nx"] + c["ny"])
    ax = 2 * crossed if c["proj"] == "Siddon" else 15 * 1.5 * crossed
    atb = 8 * vox * c["count"]
    one = es * (vox + rays)
    if c["kind"] in ("ax", "atb", "pair"):
        return {"bytes": one * (2 if c["kind"] == "pair" else 1),
                "flops": (ax if c["kind"] != "atb" else 0) + (atb if c["kind"] != "ax" else 0)}
    times = c["batch"] if c["kind"] == "autograd" else c["iters"]
    return {"bytes": 2 * one * times, "flops": (ax + atb) * times}


def tolerance(case):
    """About four times the distance from exact() that was measured over listed and drawn cases."""
    c = case
    if c["kind"] in ("ax", "atb", "pair"):
        if c["dtype"] != "f32":     # the result's rounding to its 16-bit type
            return {"rel": 6e-3 if c["dtype"] == "bf16" else 8e-4}
        return {"rel": 1e-6 if c["kind"] == "atb" else 4e-6}      # 32-bit sums over views / along rays
    if c["kind"] == "autograd":
        return {"rel": 5e-6}
    if c["kind"] == "cgls":
        return {"rel": 4e-5}        # the steps amplify the operators' rounding
    if c["kind"] == "tv":
        return {"rel": 1.3e-4}      # the gradient's direction jumps where a difference crosses 0
    if c["kind"] == "denoise":
        return {"rel": 1e-6}
    return {"rel": 1.4e-2 if c["kind"] == "unet" else 7e-3}       # BF16 activations, layer after layer
