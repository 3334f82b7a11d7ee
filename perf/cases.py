"""Performance cases: the calls a program makes of this framework, at the sizes it makes them.

A case is a dict of plain numbers and texts.  ``listed()`` are the fixed ones, ``draw(rng)``
one more of the same ranges, ``prepare`` the inputs and the plan a program keeps, ``run`` one
pass through the public entry points, ``work`` what a pass cannot do without and ``exact`` the
same outputs in 64 bits from the formulas alone (torch / numpy, none of the package's solvers).

Kinds:
  image   mask bits -> Abbe images (``Plan.intensity``), FP64 or mixed precision;
  m3d     mask bits -> amplitudes and M3D parameters (``Plan.m3d``);
  linear  mask bits + M3D parameters -> linear-model and thin-mask images (``Plan.linear``);
  socs    mask bits + M3D parameters -> STCC-SOCS images (``Plan.socs``);
  cnn     mask rasters -> M3D parameters by the six networks (``CnnPredictor.predict``);
  raster  rectangles -> packed masks with sidewall slices (``masks.rasterize``).

Images of the mixed form are kept as float32, and so are the outputs of the networks, which
are FP32 networks: that is the type the values are good to.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from euvlitho_b200 import cnn as CNN
from euvlitho_b200 import masks as MK
from euvlitho_b200.config import SimConfig, Stack
from euvlitho_b200.engine import Plan

PI = math.pi
_ABS = complex(0.95, 0.031) ** 2
_STACK = Stack(n_mo=0.924 + 0.0064j, n_si=0.999 + 0.0018j, n_ru=0.886 + 0.017j,
               d_mo=2.8, d_si=4.2, d_mosi=0.0, d_simo=0.0, d_siru=0.0, d_ru=2.5)


# ------------------------------------------------------------------ cases
def _image(name, nx, ny, box, ndivs, sources, slices, sides, refresh, pols, precision, clips,
           optics="high"):
    return dict(name=name, kind="image", nx=nx, ny=ny, box=box, ndivs=ndivs, sources=sources,
                slices=slices, sides=sides, refresh=refresh, pols=pols, precision=precision,
                clips=clips, optics=optics)


def listed():
    return [
        # one small clip, one polarisation, FP64: the interactive call (N = 121, 4 families)
        _image("image_256_fp64", 256, 256, 5, 2, 0, 1, False, False, "X", "fp64", 1),
        # small clips with the absorber as eight sidewall slices, one mask per slice
        _image("image_256_sides_mixed", 256, 256, 5, 2, 0, 8, True, False, "XY", "mixed", 2),
        # the served workload: 1024 nm clips, N = 625, 200 sources in 3 families, X + Y
        _image("image_1024_mixed", 1024, 1024, 12, 2, 200, 1, False, False, "XY", "mixed", 4),
        # the benchmark's clip (N = 961) in FP64: the accurate run of a user who checks results
        _image("image_1024_fp64", 1024, 1024, 15, 2, 200, 1, False, False, "XY", "fp64", 1),
        # the largest order box (N = 1681), eight sidewall slices, 380 sources
        _image("image_2048_sides_mixed", 2048, 2048, 20, 1, 0, 8, True, False, "XY", "mixed", 2),
        # a ragged rectangular clip whose slices each use their own 1/eps, mixed
        _image("image_ragged_refresh_mixed", 584, 424, 8, 1, 0, 3, True, True, "X", "mixed", 3),
        # the reference drivers' optics (NA 0.33, rounded diamond of orders, nine families)
        _image("image_512_reference_fp64", 512, 512, 0, 0, 0, 1, False, False, "X", "fp64", 1,
               "reference"),
        # M3D parameters for training data, FP64 (N = 2177), reference optics
        dict(name="m3d_1024_fp64", kind="m3d", nx=1024, ny=1024, clips=1),
        # linear-model and thin-mask images from M3D parameters, reference optics
        dict(name="linear_1024", kind="linear", nx=1024, ny=1024, clips=2),
        # SOCS images with resident kernels, reference optics
        dict(name="socs_1024", kind="socs", nx=1024, ny=1024, clips=4),
        # the networks on one mask (latency: the weight stream) and on a batch
        dict(name="cnn_1", kind="cnn", clips=1),
        dict(name="cnn_24", kind="cnn", clips=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["image"] * 7 + ["m3d", "linear", "socs", "cnn", "raster"])
    if kind == "cnn":
        return dict(kind="cnn", clips=_log_int(rng, 1, 24))
    if kind == "raster":
        return dict(kind="raster", nx=8 * _log_int(rng, 32, 256), ny=8 * _log_int(rng, 32, 256),
                    clips=_log_int(rng, 1, 32), slices=rng.randint(1, 8))
    if kind in ("m3d", "linear", "socs"):
        return dict(kind=kind, nx=8 * rng.randint(48, 128), ny=8 * rng.randint(48, 128),
                    clips=_log_int(rng, 1, {"m3d": 1, "linear": 2, "socs": 4}[kind]))
    if rng.random() < 0.15:
        return dict(kind="image", nx=8 * rng.randint(32, 64), ny=8 * rng.randint(32, 64), box=0,
                    ndivs=0, sources=0, slices=1, sides=False, refresh=False, pols="X",
                    precision="fp64", clips=1, optics="reference")
    precision = rng.choice(["mixed", "mixed", "fp64"])
    slices = rng.choice([1, 1, 1, 2, 3, 8])
    # the mixed form serves thick slabs up to 25 x 25 orders and thin slices beyond
    largest = 13 if precision == "fp64" else {1: 12, 8: 18}.get(slices, 11)
    top = int(largest / 0.55 * 54 / 8) - 8
    nx, ny = 8 * _log_int(rng, 32, top), 8 * _log_int(rng, 32, top)
    # the box holds every order the pupil reads, and no order near grazing
    need = max(math.ceil(0.55 * nx / 4 / 13.5), math.ceil(0.55 * ny / 8 / 13.5))
    box = max(5, need + rng.randint(1, 3))
    box = max(min(box, int(min(nx, ny) * 0.033), largest), need)
    sides = slices > 1 and rng.random() < 0.7
    refresh = 1 < slices < 8 and rng.random() < 0.5
    ndivs = rng.choice([1, 2]) if min(nx, ny) <= 1024 else 1
    pols = rng.choice(["X", "Y", "XY"])
    per_clip = (2 * box + 1) ** 6 * slices * len(pols) * ndivs * ndivs
    budget = 1681 ** 3 * 8 * 2 * 2 // (2 if precision == "mixed" else 12)
    clips = max(1, min(rng.randint(1, 6), budget // per_clip))
    return dict(kind="image", nx=nx, ny=ny, box=box, ndivs=ndivs,
                sources=rng.choice([0, 0, 50, 120]), slices=slices, sides=sides, refresh=refresh,
                pols=pols, precision=precision, clips=clips, optics="high")


# ------------------------------------------------------------------ inputs
def _config(case):
    if case["kind"] in ("m3d", "linear", "socs") or case["optics"] == "reference":
        return SimConfig(ndivx=case["nx"], ndivy=case["ny"])
    n = case["slices"]
    return SimConfig(ndivx=case["nx"], ndivy=case["ny"], na=0.55, mx=4, my=8, theta0=-6.0,
                     stack=_STACK, eabs=(_ABS,) * n, dabs=(60.0 / n,) * n, sigma1=0.9,
                     sigma2=0.5, illum_type=1, order_kind="box", lbox=case["box"],
                     mbox=case["box"], ndivs=case["ndivs"], max_sources=case["sources"] or None,
                     refresh_sigma=case["refresh"])


def _layout(rng, nx, ny):
    """Lines 16-64 nm wide at a pitch of 2-4 widths, and square contacts, until about 36 % of
    the clip is absorber: rectangles (x0, x1, y0, y1)."""
    rects = []
    w = rng.randint(16, 48)
    pitch = int(w * rng.uniform(2.5, 4.0))
    vertical = rng.random() < 0.5
    n = nx if vertical else ny
    for s in range(rng.randrange(pitch), n, pitch):
        rects.append((s, min(s + w, n), 0, ny) if vertical else (0, nx, s, min(s + w, n)))
    area = w / pitch
    while area < 0.40:
        c = rng.randint(16, 64)
        x, y = rng.randrange(max(1, nx - c)), rng.randrange(max(1, ny - c))
        rects.append((x, min(x + c, nx), y, min(y + c, ny)))
        area += c * c / (nx * ny) * (1 - area)
    return rects


def _pack(absorber):
    bits = (~absorber).reshape(absorber.shape[0], -1, 8).to(torch.uint8)
    w = torch.tensor([128, 64, 32, 16, 8, 4, 2, 1], dtype=torch.uint8, device=bits.device)
    return (bits * w).sum(-1, dtype=torch.uint8)


def _masks(nx, ny, clips, slices, seed):
    """Packed masks [clips, slices, bytes] on the GPU: the drawn absorber is the bottom slice,
    the others are eroded as an 84 degree sidewall."""
    rng = random.Random("masks %d" % seed)
    out = []
    bias = 60.0 / max(slices, 1) * math.tan(math.radians(6.0))
    for _ in range(clips):
        m = np.zeros((ny, nx), bool)
        for x0, x1, y0, y1 in _layout(rng, nx, ny):
            m[y0:y1, x0:x1] = True
        a = torch.from_numpy(m).cuda()
        at, per = 0, {}
        for s in range(slices - 1, -1, -1):
            r = int(round((slices - 1 - s) * bias))
            while at < r:
                a = (a & a.roll(1, 0) & a.roll(-1, 0) & a.roll(1, 1) & a.roll(-1, 1))
                at += 1
            per[s] = a
        out.append(_pack(torch.stack([per[s] for s in range(slices)])))
    return torch.stack(out)


def _parameters(clips, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn((clips, n), dtype=torch.complex128, device="cuda", generator=g) * 1e-3
            for _ in range(3)]


N_OUTS = (1901, 1901, 1749, 1749, 1749, 1749)
CHANNELS = (1, 16, 32, 64, 128, 256)


def _network(i, seed):
    """State dict of network i with default-scale random weights."""
    g = torch.Generator(device="cuda").manual_seed(1000 * seed + i)

    def u(shape, fan):
        return (torch.rand(shape, generator=g, device="cuda") * 2 - 1) / math.sqrt(fan)

    sd = {}
    for l in range(5):
        ci, co = CHANNELS[l], CHANNELS[l + 1]
        sd["conv%d.weight" % (l + 1)] = u((co, ci, 3, 3), 9 * ci)
        sd["conv%d.bias" % (l + 1)] = u((co,), 9 * ci)
        sd["norm%d.weight" % (l + 1)] = 1 + 0.2 * torch.randn(co, generator=g, device="cuda")
        sd["norm%d.bias" % (l + 1)] = 0.2 * torch.randn(co, generator=g, device="cuda")
        sd["norm%d.running_mean" % (l + 1)] = 0.2 * torch.randn(co, generator=g, device="cuda")
        sd["norm%d.running_var" % (l + 1)] = 0.5 + torch.rand(co, generator=g, device="cuda")
    sd["fc1.weight"] = u((4096, 65536), 65536)
    sd["fc1.bias"] = u((4096,), 65536)
    sd["fc2.weight"] = u((N_OUTS[i], 4096), 4096)
    sd["fc2.bias"] = u((N_OUTS[i],), 4096)
    return sd


def _factors(seed):
    g = np.random.default_rng(seed)
    f0, fx, fy = (0.5 + g.random(n) for n in (N_OUTS[0], N_OUTS[2], N_OUTS[4]))
    return [f0, f0, fx, fx, fy, fy]


def _rectangles(case, seed):
    rng = random.Random("raster %d" % seed)
    return [_layout(rng, case["nx"], case["ny"]) for _ in range(case["clips"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "raster":
        er = MK.sidewall_erosion(case["slices"], 60.0 / case["slices"])
        return dict(case=case, rects=_rectangles(case, seed), erosion=er)
    if kind == "cnn":
        pred = CNN.CnnPredictor([_network(i, 1) for i in range(6)], _factors(1))
        torch.cuda.empty_cache()
        pred.workspace(case["clips"])
        bits = _masks(2048, 2048, case["clips"], 1, seed)[:, 0].contiguous()
        return dict(case=case, predictor=pred, bits=bits)
    cfg = _config(case)
    state = dict(case=case)
    if kind == "image":
        slices = case["slices"] if case["sides"] else 1
        plan = Plan(cfg, precision=case["precision"], pols=tuple(case["pols"]))
        plan.intensity_batch(case["clips"], slices)
        state["masks"] = _masks(case["nx"], case["ny"], case["clips"], slices, seed)
    else:
        plan = Plan(cfg)
        state["masks"] = _masks(case["nx"], case["ny"], case["clips"], 1, seed)[:, 0].contiguous()
        if kind == "m3d":
            plan.m3d_tables()
        elif kind == "linear":
            plan.linear_tables()
        else:
            plan.socs_tables()
        if kind != "m3d":
            state["parameters"] = _parameters(case["clips"], plan.ncut, seed)
    state["plan"] = plan
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "image":
        img = state["plan"].intensity(state["masks"])
        return img if case["precision"] == "fp64" else img.to(torch.float32)
    if kind == "m3d":
        r = state["plan"].m3d(state["masks"])
        return {k: r[k] for k in ("a0", "ax", "ay", "Ax")}
    if kind == "linear":
        lin, thin = state["plan"].linear(state["masks"], *state["parameters"])
        return [lin, thin]
    if kind == "socs":
        return state["plan"].socs(state["masks"], *state["parameters"])
    if kind == "cnn":
        return [a.astype(np.float32) for a in state["predictor"].predict(state["bits"])]
    return MK.rasterize(state["rects"], case["nx"], case["ny"], state["erosion"])


# ------------------------------------------------------------------ the optics in numbers
class _Optics:
    """Order, pupil and source sets of a configuration, from its constants."""

    def __init__(self, c):
        self.c = c
        self.k = 2 * PI / c.wavelength
        self.dx, self.dy = float(c.ndivx), float(c.ndivy)
        self.gx, self.gy = 2 * PI / self.dx, 2 * PI / self.dy
        self.kx0 = self.k * math.sin(math.radians(c.theta0)) * math.cos(PI / 180 * (90.0 - c.azimuth))
        self.ky0 = self.k * math.sin(math.radians(c.theta0)) * math.sin(PI / 180 * (90.0 - c.azimuth))
        self.z0 = sum(c.dabs) + c.z0_offset
        self.xd, self.yd = c.ndivx // c.mx, c.ndivy // c.my
        rx, ry = c.na * self.dx / c.mx / c.wavelength, c.na * self.dy / c.my / c.wavelength
        self.ls, self.ms = int(rx + 1), int(ry + 1)
        self.lp, self.mp = int(2 * rx + 1e-4), int(2 * ry + 1e-4)
        if c.order_kind == "box":
            self.L, self.M = c.lbox, c.mbox
        else:
            self.L, self.M = int(rx * c.cut), int(ry * c.cut)
        l, m = np.meshgrid(np.arange(-self.L, self.L + 1), np.arange(-self.M, self.M + 1),
                           indexing="ij")
        keep = np.ones(l.shape, bool)
        if c.order_kind == "diamond":
            keep = (abs(l) / (self.L + 0.01) + 1) * (abs(m) / (self.M + 0.01) + 1) <= 2.0
        self.l, self.m = l[keep], m[keep]
        self.pos = np.full((2 * self.L + 1, 2 * self.M + 1), -1)
        self.pos[self.l + self.L, self.m + self.M] = np.arange(self.l.size)
        sl, sm = np.meshgrid(np.arange(-self.ls, self.ls + 1), np.arange(-self.ms, self.ms + 1),
                             indexing="ij")
        ok = self.in_na(sl, sm)
        self.na_l, self.na_m = sl[ok], sm[ok]
        pl, pm = np.meshgrid(np.arange(-self.lp, self.lp + 1), np.arange(-self.mp, self.mp + 1),
                             indexing="ij")
        seen = np.array([[self.in_na(a + self.na_l, b + self.na_m).sum() for a, b in zip(ra, rb)]
                         for ra, rb in zip(pl, pm)])
        self.pl, self.pm = pl[seen > 0], pm[seen > 0]
        self.full = seen[seen > 0] >= 8

    def in_na(self, l, m):
        c = self.c
        return (l * c.mx / self.dx) ** 2 + (m * c.my / self.dy) ** 2 <= (c.na / c.wavelength) ** 2

    def annulus(self, kx, ky):
        c = self.c
        r = np.hypot(kx * c.mx, ky * c.my)
        return (r <= self.k * c.na * c.sigma1) & (r >= self.k * c.na * c.sigma2)

    def families(self):
        c = self.c
        nd = c.ndivs or max(1, int(180.0 / PI * c.wavelength / self.dx / c.sigmadiv))
        lm = int(self.k * c.na / c.mx * c.sigma1 / self.gx + 1)
        mm = int(self.k * c.na / c.my * c.sigma1 / self.gy + 1)
        l, m = np.meshgrid(np.arange(-lm, lm + 1), np.arange(-mm, mm + 1), indexing="ij")
        l, m = l.ravel(), m.ravel()
        left, out = c.max_sources or 10 ** 9, []
        for ix in range(nd):
            for iy in range(nd):
                ox, oy = self.gx * ix / nd, self.gy * iy / nd
                ok = np.nonzero(self.annulus(l * self.gx + ox, m * self.gy + oy))[0][:left]
                left -= ok.size
                if ok.size:
                    out.append((ox, oy, l[ok], m[ok]))
        return out

    def grid_sources(self, mesh=0.2):
        c = self.c
        s = self.k * mesh * PI / 180
        lm = int(self.k * c.na / c.mx * c.sigma1 / s) + 1
        mm = int(self.k * c.na / c.my * c.sigma1 / s) + 1
        l, m = np.meshgrid(np.arange(-lm, lm + 1), np.arange(-mm, mm + 1), indexing="ij")
        kx, ky = (l * s).ravel(), (m * s).ravel()
        ok = self.annulus(kx, ky)
        return kx[ok], ky[ok]

    def pupil(self, kx, ky, z=0.0):
        """Inside the pupil, phase and polarisation columns R[..., 3, 2] at mask-side (kx, ky)."""
        c, k = self.c, self.k
        p2 = (c.mx * kx) ** 2 + (c.my * ky) ** 2
        inside = p2 <= (c.na * k) ** 2
        phase = np.exp(1j * ((kx + self.kx0) ** 2 + (ky + self.ky0) ** 2) / 2 / k * self.z0
                       + 1j * p2 / 2 / k * z)
        one = np.ones_like(kx)
        zero = np.zeros_like(kx)
        s0 = np.stack([self.kx0 * one, self.ky0 * one,
                       -math.sqrt(k * k - self.kx0 ** 2 - self.ky0 ** 2) * one], -1)
        p = np.stack([kx, ky, zero], -1)
        pp = np.stack([c.mx * kx, c.my * ky, -np.sqrt(np.maximum(k * k - p2, 0.0))], -1)
        ez = np.stack([zero, zero, one], -1)

        def unit(v):
            n = np.linalg.norm(v, axis=-1, keepdims=True)
            return v / np.where(n == 0, 1.0, n)

        far = (kx * kx + ky * ky > 1e-5)[..., None]
        es = np.where(far, unit(np.cross(p, s0)), unit(np.cross(ez, s0)))
        esp = np.where(far, unit(np.cross(pp, ez)), -es)
        em = np.where(far, np.cross(es, unit(p + s0)), np.cross(es, s0) / k)
        emp = np.where(far, np.cross(esp, pp) / k, np.cross(esp, -ez))
        R = esp[..., :, None] * es[..., None, :2] + emp[..., :, None] * em[..., None, :2]
        return inside, phase, R


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _absorber(bits, nx, ny):
    """Absorber indicator [x][y], y up, of one packed mask."""
    b = (bits[:, None] >> torch.arange(7, -1, -1, device=bits.device, dtype=torch.uint8)) & 1
    return (1 - b.reshape(ny, nx).double()).flip(0).T


def _spectrum(pattern, L, M):
    nx, ny = pattern.shape
    F = torch.fft.fft2(pattern.to(torch.complex128)) / (nx * ny)
    return F[torch.arange(-L, L + 1) % nx][:, torch.arange(-M, M + 1) % ny]


def _stack_fields(o, pol, kx, ky):
    """(U_down, U_up) on top of the multilayer and the capping layer's wave number, per order."""
    st, k = o.c.stack, o.k
    e = {"mo": st.n_mo ** 2, "si": st.n_si ** 2, "ru": st.n_ru ** 2, "ms": st.n_mosi2 ** 2,
         "rs": st.n_rusi ** 2, "sub": st.n_sio2 ** 2}
    kp = kx if pol == "X" else ky
    al = {n: np.sqrt(k * k * v - kx * kx - ky * ky + 0j) for n, v in e.items()}
    b = {n: k - kp * kp / k / v for n, v in e.items()}

    def layer(below, n, d):
        cj, a, x = b[below] / b[n], al[below] / al[n], np.exp(1j * al[n] * d)
        return 0.5 * (cj + a) / x, 0.5 * (cj - a) / x, 0.5 * (cj - a) * x, 0.5 * (cj + a) * x

    def step(T, u, v):
        return T[0] * u + T[1] * v, T[2] * u + T[3] * v

    u, _, v, _ = layer("sub", "mo", st.d_mo)
    for i in range(st.nml - 1, -1, -1):
        if i < st.nml - 1:
            u, v = step(layer("ms", "mo", st.d_mo), u, v)
        u, v = step(layer("mo", "ms", st.d_mosi), u, v)
        u, v = step(layer("ms", "si", st.d_si), u, v)
        u, v = step(layer("si", "ms", st.d_simo) if i else layer("si", "rs", st.d_siru), u, v)
    u, v = step(layer("rs", "ru", st.d_ru), u, v)
    return u, v, al["ru"], 1j * b["ru"]


def _cos_sinc(D, d, a, R):
    """cos(sqrt(D) d) and sin(sqrt(D) d) / sqrt(D): Taylor series about a * I, coefficients
    from samples on the circle of radius R."""
    n = D.shape[0]
    z = np.sqrt(a + R * np.exp(2j * PI * np.arange(256) / 256))
    cs = [np.fft.fft(f) / 256 for f in (np.cos(z * d), np.sin(z * d) / z)]
    eye = torch.eye(n, dtype=torch.complex128, device=D.device)
    E = (D - a * eye) / R
    # up to the first coefficients below the samples' own rounding
    top = next(i for i in range(128) if all(abs(c[i]) < 1e-15 * abs(c).max() for c in cs))
    out = []
    for c in cs:
        p = eye * complex(c[top])
        for i in range(top - 1, -1, -1):
            p = p @ E
            p.diagonal().add_(complex(c[i]))
        out.append(p)
    return out


def _amplitudes(o, pol, ox, oy, spectra, l, m, L, M, sl, sm):
    """Reflected amplitudes [N][sources] of one incidence: l, m the orders, spectra one
    absorber spectrum per slice, sl, sm the source orders."""
    c, k = o.c, o.k
    kx, ky = o.kx0 + ox + o.gx * l, o.ky0 + oy + o.gy * m
    kxy2 = kx * kx + ky * ky
    klm = _t(np.sqrt(k * k - kxy2)).to(torch.complex128)
    u, v, alru, bru = _stack_fields(o, pol, kx, ky)
    kp = kx if pol == "X" else ky
    tkx, tky, tkp = _t(kx), _t(ky), _t(kp)
    dl, dm = _t(l[:, None] - l[None, :]), _t(m[:, None] - m[None, :])
    eye = torch.eye(l.size, dtype=torch.complex128, device="cuda")
    X = Y = Gup = None
    for n in range(c.nabs - 1, -1, -1):
        e, d = complex(c.eabs[n]), float(c.dabs[n])
        F = spectra[n][dl + 2 * L, dm + 2 * M]
        zero = ((dl == 0) & (dm == 0)).to(torch.complex128)
        leps = np.log(e) * F
        D = k * k * ((e - 1) * F + zero)
        D = D + (o.gx * dl.double() * tkx if pol == "X" else o.gy * dm.double() * tky) * leps
        D.diagonal().sub_(_t(kxy2))
        if Gup is None or c.refresh_sigma:
            G = 1j * (k * eye - tkp[:, None] / k * ((1 / e - 1) * F + zero) * tkp[None, :])
        if Gup is None:
            Z = torch.linalg.solve(G, torch.diag(_t(bru * (u + v))))
            Y2 = torch.diag(_t(alru * (u - v)))
        else:
            Z = torch.linalg.solve(G, Gup @ X) if c.refresh_sigma else X
            Y2 = Y
        a = k * k * (1 + (e - 1) / 2) - 0.5 * (kxy2.max() + kxy2.min())
        R = 1.5 * (k * k * abs(e - 1) / 2 + 0.5 * (kxy2.max() - kxy2.min()))
        C, S = _cos_sinc(D, d, a, R)
        X, Y, Gup = C @ Z - 1j * (S @ Y2), C @ Y2 - 1j * (D @ (S @ Z)), G
    col = np.array([int(np.nonzero((l == a) & (m == b))[0][0]) for a, b in zip(sl, sm)])
    kz2 = 2 * np.sqrt(k * k - (o.kx0 + ox + o.gx * sl) ** 2 - (o.ky0 + oy + o.gy * sm) ** 2)
    rhs = torch.zeros((l.size, col.size), dtype=torch.complex128, device="cuda")
    rhs[_t(col), torch.arange(col.size, device="cuda")] = _t(kz2).to(torch.complex128)
    A = -(Y @ torch.linalg.solve(klm[:, None] * X + Y, rhs)) / klm[:, None]
    A[_t(col), torch.arange(col.size, device="cuda")] += 1.0
    return A


def _image_of(o, fields):
    """Sum over sources of |E|^2 on the image grid; fields [S][3][pupil] on (pl, pm)."""
    img = torch.zeros((o.xd, o.yd), dtype=torch.float64, device="cuda")
    ix, iy = _t(o.pl % o.xd), _t(o.pm % o.yd)
    for s in range(0, fields.shape[0], 32):
        f = fields[s:s + 32]
        g = torch.zeros((f.shape[0], 3, o.xd, o.yd), dtype=torch.complex128, device="cuda")
        g[:, :, ix, iy] = f
        g = torch.fft.ifft2(g, norm="forward")
        img += (g.real ** 2 + g.imag ** 2).sum((0, 1))
    return img


def _exact_image(case, seed):
    o = _Optics(_config(case))
    c, k = o.c, o.k
    slices = case["slices"] if case["sides"] else 1
    masks = _masks(case["nx"], case["ny"], case["clips"], slices, seed)
    fams = o.families()
    total = sum(f[2].size for f in fams)
    out = torch.zeros((case["clips"], len(case["pols"]), o.xd, o.yd), dtype=torch.float64,
                      device="cuda")
    for ci in range(case["clips"]):
        spec = [_spectrum(_absorber(masks[ci, s], case["nx"], case["ny"]), 2 * o.L, 2 * o.M)
                for s in range(slices)]
        spec = spec if slices > 1 else spec * c.nabs
        for pi, pol in enumerate(case["pols"]):
            for ox, oy, sl, sm in fams:
                A = _amplitudes(o, pol, ox, oy, spec, o.l, o.m, o.L, o.M, sl, sm)
                kxn = ox + o.gx * (sl[:, None] + o.pl[None, :])
                kyn = oy + o.gy * (sm[:, None] + o.pm[None, :])
                inside, phase, R = o.pupil(kxn, kyn, float(c.z))
                L, M = sl[:, None] + o.pl[None, :], sm[:, None] + o.pm[None, :]
                idx = np.where(inside, o.pos[np.clip(L + o.L, 0, 2 * o.L),
                                             np.clip(M + o.M, 0, 2 * o.M)], 0)
                k1 = (o.kx0 + ox + o.gx * sl) if pol == "X" else (o.ky0 + oy + o.gy * sm)
                f = 1j * k / np.sqrt(k * k - k1 * k1)[:, None] * phase * inside
                f = f[:, None, :] * np.moveaxis(R[..., 0 if pol == "X" else 1], -1, 1)
                a = A.T[torch.arange(sl.size, device="cuda")[:, None], _t(idx)]
                out[ci, pi] += _image_of(o, _t(f) * a[:, None, :]) / total
    return out


def _uniform(o):
    """Amplitudes of the all-vacuum and the all-absorber mask at every NA source order
    (diagonal problems), in the order of na_l, na_m, X polarisation."""
    n = o.na_l.size
    res = []
    for dc in (0.0, 1.0):
        L, M = int(abs(o.na_l).max()), int(abs(o.na_m).max())
        F = torch.zeros((4 * L + 1, 4 * M + 1), dtype=torch.complex128, device="cuda")
        F[2 * L, 2 * M] = dc
        A = _amplitudes(o, "X", 0.0, 0.0, [F] * o.c.nabs, o.na_l, o.na_m, L, M, o.na_l, o.na_m)
        res.append(A.diagonal().cpu().numpy()[:n])
    return res


def _exact_m3d(case, seed):
    o = _Optics(_config(case))
    masks = _masks(case["nx"], case["ny"], case["clips"], 1, seed)
    vc, ab = _uniform(o)
    centre = int(np.nonzero((o.na_l == 0) & (o.na_m == 0))[0][0])
    keep = {"a0": [], "ax": [], "ay": [], "Ax": []}
    for ci in range(case["clips"]):
        pattern = _absorber(masks[ci, 0], case["nx"], case["ny"])
        spec = _spectrum(pattern, 2 * o.L, 2 * o.M)
        A = _amplitudes(o, "X", 0.0, 0.0, [spec] * o.c.nabs, o.l, o.m, o.L, o.M, o.na_l, o.na_m)
        F = _spectrum(1 - pattern, o.lp, o.mp).cpu().numpy()
        An = A.cpu().numpy()
        thin = _thin(o, F, vc[centre], ab[centre])
        res = np.zeros((3, o.pl.size), np.complex128)
        for n, (p, q) in enumerate(zip(o.pl, o.pm)):
            s = np.nonzero(o.in_na(o.na_l + p, o.na_m + q))[0]
            i = o.pos[o.na_l[s] + p + o.L, o.na_m[s] + q + o.M]
            f = An[i, s] / (vc[s] / abs(vc[s])) - thin[n]
            if o.full[n]:
                B = np.stack([np.ones(s.size), o.na_l[s] + p / 2, o.na_m[s] + q / 2], 1)
                res[:, n] = np.linalg.solve(B.T @ B, B.T @ f)
            else:
                res[0, n] = f.mean()
        for key, v in zip(("a0", "ax", "ay"), res):
            keep[key].append(_t(v))
        keep["Ax"].append(A.T)
    return {key: torch.stack(v) for key, v in keep.items()}


def _thin(o, F, vc, ab):
    """Thin-mask amplitude per pupil point, phase of the vacuum reflection taken out."""
    kxp, kyp = o.gx * o.pl, o.gy * o.pm
    ph = np.exp(-1j * (o.kx0 * kxp + kxp ** 2 / 2 + o.ky0 * kyp + kyp ** 2 / 2) / o.k * o.z0)
    f = (vc - ab) * F[o.pl + o.lp, o.pm + o.mp] * ph + ab * ((o.pl == 0) & (o.pm == 0))
    return f / (vc / abs(vc))


def _exact_linear(case, seed):
    o = _Optics(_config(case))
    masks = _masks(case["nx"], case["ny"], case["clips"], 1, seed)
    par = _parameters(case["clips"], o.pl.size, seed)
    vc, ab = _uniform(o)
    cn = int(np.nonzero((o.na_l == 0) & (o.na_m == 0))[0][0])
    kx, ky = o.grid_sources()
    inside, phase, R = o.pupil(kx[:, None] + o.gx * o.pl, ky[:, None] + o.gy * o.pm, float(o.c.z))
    f = 1j * o.k / np.sqrt(o.k ** 2 - (o.kx0 + kx) ** 2)[:, None] * phase * inside
    f = _t(f[:, None, :] * np.moveaxis(R[..., 0], -1, 1))
    lin, flat = [], []
    ls, ms = _t(kx / o.gx)[:, None] + _t(o.pl / 2), _t(ky / o.gy)[:, None] + _t(o.pm / 2)
    for ci in range(case["clips"]):
        F = _spectrum(1 - _absorber(masks[ci, 0], case["nx"], case["ny"]), o.lp, o.mp)
        thin = _t(_thin(o, F.cpu().numpy(), vc[cn], ab[cn]))
        full = thin + par[0][ci] + par[1][ci] * ls + par[2][ci] * ms
        lin.append(_image_of(o, f * full[:, None, :]) / kx.size)
        flat.append(_image_of(o, f * thin[None, None, :]) / kx.size)
    return [torch.stack(lin), torch.stack(flat)]


def _exact_socs(case, seed, keep=100, keep_xy=20, grid=64):
    o = _Optics(_config(case))
    masks = _masks(case["nx"], case["ny"], case["clips"], 1, seed)
    par = _parameters(case["clips"], o.pl.size, seed)
    vc, ab = _uniform(o)
    cn = int(np.nonzero((o.na_l == 0) & (o.na_m == 0))[0][0])
    kx, ky = o.grid_sources()
    inside, phase, R = o.pupil(o.gx * o.pl[:, None] + kx, o.gy * o.pm[:, None] + ky, float(o.c.z))
    P = [_t(phase * inside * R[..., i, 0]) for i in range(3)]
    w0 = _t(o.k ** 2 / (o.k ** 2 - (o.kx0 + kx) ** 2))
    # the point (0, 0) counts once per order of the wide set beyond the pupil points
    z = int(np.nonzero((o.pl == 0) & (o.pm == 0))[0][0])
    copies = math.sqrt(1.0 + max(0, o.l.size - o.pl.size))
    eig = []
    for w in (w0, _t(kx) * w0, _t(ky) * w0):
        T = sum((p * w) @ p.conj().T for p in P) / kx.size
        T[z, :] *= copies
        T[:, z] *= copies
        a, v = torch.linalg.eigh((T + T.conj().T) / 2)
        v[z, :] /= copies
        best = torch.argsort(-a.abs(), stable=True)
        eig.append((a[best], v[:, best].T))
    ix, iy = _t(o.pl % grid), _t(o.pm % grid)

    def field(v):
        g = torch.zeros((v.shape[0], grid, grid), dtype=torch.complex128, device="cuda")
        g[:, ix, iy] = v
        return torch.fft.ifft2(g, norm="forward")

    out = []
    h = grid // 2
    for ci in range(case["clips"]):
        F = _spectrum(1 - _absorber(masks[ci, 0], case["nx"], case["ny"]), o.lp, o.mp)
        A0 = _t(_thin(o, F.cpu().numpy(), vc[cn], ab[cn])) + par[0][ci]
        ax, ay = par[1][ci], par[2][ci]
        (a0, p0), (a1, p1), (a2, p2) = eig
        f0 = field(A0 * p0[:keep])
        small = (a0[:keep, None, None] * f0.abs() ** 2).sum(0)
        for f, b, g in ((field(A0 * p1[:keep_xy]), a1, field(ax / o.gx * p1[:keep_xy])),
                        (field(A0 * p2[:keep_xy]), a2, field(ay / o.gy * p2[:keep_xy])),
                        (f0[:keep_xy], a0,
                         field((ax * _t(o.pl / 2) + ay * _t(o.pm / 2)) * p0[:keep_xy]))):
            small = small + (2 * b[:keep_xy, None, None] * (f * g.conj()).real).sum(0)
        s = torch.fft.fft2(small.to(torch.complex128), norm="forward")
        big = torch.zeros((o.xd, o.yd), dtype=torch.complex128, device="cuda")
        i = torch.arange(-h, h, device="cuda")
        big[(i % o.xd)[:, None], (i % o.yd)[None, :]] = s[(i % grid)[:, None], (i % grid)[None, :]]
        out.append(torch.fft.ifft2(big, norm="forward").real)
    return torch.stack(out)


def _exact_cnn(case, seed):
    bits = _masks(2048, 2048, case["clips"], 1, seed)[:, 0]
    fac = _factors(1)
    shifts = torch.arange(7, -1, -1, device="cuda", dtype=torch.uint8)
    x0 = torch.stack([((b[:, None] >> shifts) & 1).reshape(512, 4, 512, 4).double().mean((1, 3))
                      for b in bits])[:, None]
    out = []
    for i in range(6):
        sd = {k: v.double() for k, v in _network(i, 1).items()}
        rows = []
        for s in range(0, x0.shape[0], 4):
            x = x0[s:s + 4]
            for l in range(1, 6):
                x = torch.nn.functional.pad(x, (1, 1, 1, 1), mode="circular")
                x = torch.nn.functional.conv2d(x, sd["conv%d.weight" % l], sd["conv%d.bias" % l])
                x = torch.nn.functional.max_pool2d(x.relu(), 2)
                x = torch.nn.functional.batch_norm(
                    x, sd["norm%d.running_mean" % l], sd["norm%d.running_var" % l],
                    sd["norm%d.weight" % l], sd["norm%d.bias" % l], False, 0.0, 1e-5)
            x = (x.flatten(1) @ sd["fc1.weight"].T + sd["fc1.bias"]).relu()
            rows.append(x @ sd["fc2.weight"].T + sd["fc2.bias"])
        out.append(torch.cat(rows).cpu().numpy() / fac[i])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "raster":
        return None
    return {"image": _exact_image, "m3d": _exact_m3d, "linear": _exact_linear,
            "socs": _exact_socs, "cnn": _exact_cnn}[kind](case, seed)


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: inputs and outputs once (and the network weights).  Operations of an image: per
    unit and slice three complex N^3 products (the slab's two functions and their use), one
    complex factorisation and the solve per unit, and the Fourier sums of the image."""
    kind = case["kind"]
    if kind == "raster":
        n = case["nx"] * case["ny"] // 8 * case["clips"] * case["slices"]
        return {"bytes": n, "flops": 0}
    if kind == "cnn":
        conv = sum(2.0 * (512 >> l) ** 2 * CHANNELS[l + 1] * 9 * CHANNELS[l] for l in range(5))
        fc = sum(65536 * 4096 + 4096 * n for n in N_OUTS)
        return {"bytes": 4.0 * fc + case["clips"] * (2048 * 2048 / 8 + 8.0 * sum(N_OUTS)),
                "flops": case["clips"] * (6 * conv + 2.0 * fc)}
    o = _Optics(_config(case))
    clips = case["clips"]
    mask = clips * case["nx"] * case["ny"] / 8
    image = o.xd * o.yd
    fft = 5.0 * image * math.log2(max(2, image))

    def solve(n, slices, sources):
        return 24.0 * n ** 3 * slices + 8.0 / 3 * n ** 3 + 8.0 * n * n * sources

    if kind == "image":
        fams = o.families()
        slices = case["slices"]
        pols = len(case["pols"])
        flops = sum(solve(o.l.size, slices, f[2].size) + f[2].size * 3 * fft for f in fams)
        out = clips * pols * image * (8 if case["precision"] == "fp64" else 4)
        return {"bytes": mask * (slices if case["sides"] else 1) + out,
                "flops": clips * pols * flops}
    if kind == "m3d":
        s = o.na_l.size
        return {"bytes": mask + clips * 16.0 * (s * o.l.size + 3 * o.pl.size),
                "flops": clips * solve(o.l.size, o.c.nabs, s)}
    if kind == "linear":
        s = o.grid_sources()[0].size
        return {"bytes": mask + clips * (48.0 * o.pl.size + 16.0 * image),
                "flops": clips * 2 * s * 3 * fft}
    return {"bytes": mask + clips * (48.0 * o.pl.size + 8.0 * image) + 16.0 * 140 * o.pl.size,
            "flops": clips * (200 * 5.0 * 64 * 64 * 12 + fft)}
