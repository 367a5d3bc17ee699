"""The workloads this package is timed on: one entry per way a program uses it.

``listed()`` names twelve of them, ``draw(rng)`` gives another of the same ranges.  ``prepare`` makes
the inputs (on the GPU, from the seed alone) and the plan a program keeps, ``run`` is one pass through
the public entry points, ``work`` the bytes and operations of a pass that no implementation can avoid,
and ``exact`` the same result in 64-bit torch, written here from the definitions.

Array order is the package's: sinogram (na, nb), projections (na, nt, ns), image ([nz,] ny, nx).
"""
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "sinograms.jl_gb300"))

import sinograms as S  # noqa: E402
from sinograms import learned  # noqa: E402

# --------------------------------------------------------------------------------- the cases
#
# Fields: path (fbp, fdk, batch, dd, sf, net, grad); kind of detector; nb/na, ns/nt/na; nx/ny/nz;
# d (bin), dx (pixel; 0: the image square inscribed in the field of view), orbit in degrees (0: short
# scan), offset of the detector in bins, window, slices of a stack, storage form of the projections.

_GE = dict(d=1.0239, dsd=949.075, dod=408.075)  # the fan-beam scanner of the package's presets


def listed():
    return [
        # a thumbnail of one slice: the smallest call, all launch and host latency; odd sizes
        dict(name="fbp flat 97x61 to 65x63", path="fbp", kind="flat", nb=97, na=61, nx=65, ny=63, d=1.0, dx=0.0,
             orbit=360.0, offset=0.0, window="none", slices=1, dsd=400.0, dod=150.0),
        # one parallel-beam slice, apodised: an ordinary interactive call
        dict(name="fbp par 256x180 hann", path="fbp", kind="par", nb=256, na=180, nx=256, ny=256, d=1.0, dx=1.0,
             orbit=180.0, offset=0.0, window="hann", slices=1, dsd=0.0, dod=0.0),
        # one slice of a short scan (Parker weights) with noise, at diagnostic size
        dict(name="fbp arc short 888x512", path="fbp", kind="arc", nb=888, na=512, nx=512, ny=512, dx=0.9766,
             orbit=0.0, offset=0.0, window="none", slices=1, **_GE),
        # a stack of slices of the full-rotation preset (quarter detector offset): throughput
        dict(name="fbp arc 888x984 stack of 8", path="fbp", kind="arc", nb=888, na=984, nx=512, ny=512, dx=0.9766,
             orbit=360.0, offset=1.25, window="none", slices=8, **_GE),
        # a small cone-beam volume of odd sizes from a short scan on a curved detector
        dict(name="fdk arc short 301x123x200", path="fdk", kind="arc", ns=301, nt=123, na=200, nx=197, ny=211, nz=101,
             ds=1.0, dx=0.0, orbit=0.0, offset=0.25, window="hann", storage="f32", dsd=1000.0, dod=400.0),
        # the cone-beam volume of the package's benchmark, in full precision and in the FP16 form
        dict(name="fdk flat 512 f32", path="fdk", kind="flat", ns=512, nt=384, na=720, nx=512, ny=512, nz=256, ds=1.0,
             dx=0.5, orbit=360.0, offset=0.0, window="none", storage="f32", dsd=1000.0, dod=400.0),
        dict(name="fdk flat 512 f16", path="fdk", kind="flat", ns=512, nt=384, na=720, nx=512, ny=512, nz=256, ds=1.0,
             dx=0.5, orbit=360.0, offset=0.0, window="none", storage="f16", dsd=1000.0, dod=400.0),
        # a night's queue of uneven cone-beam scans (the seeded generator of the batched workload)
        dict(name="batch of 6 f16", path="batch", scans=6, geometry_seed=4, storage="f16"),
        # one iteration of an iterative solver on the sparse-view scan: forward and back, in either model
        dict(name="dd pair arc 888x90", path="dd", kind="arc", nb=888, na=90, nx=512, dx=0.9766, **_GE),
        dict(name="sf pair arc 888x90", path="sf", kind="arc", nb=888, na=90, nx=512, ny=512, dx=0.9766, orbit=360.0,
             offset=0.0, **_GE),
        # sparse-view reconstruction through the learned row filter
        dict(name="learned fbp 888x90", path="net", kind="arc", nb=888, na=90, nx=512, ny=512, dx=0.9766,
             orbit=360.0, offset=0.0, window="none", slices=1, **_GE),
        # the learned filter's loss and gradients on a training batch
        dict(name="learned grad 4096x888", path="grad", rows=4096, nb=888),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _views(rng, lo, hi):
    """Scans come with round numbers of views as often as not."""
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.5 else max(10, n // 10 * 10)


def _scanner(rng, n):
    """Source and detector distances for n bins of 1 mm: fans of 20 to 55 degrees."""
    dsd = round(n / (2 * math.tan(math.radians(rng.uniform(20, 55)) / 2)), 1)
    return dict(dsd=dsd, dod=round(rng.uniform(0.3, 0.45) * dsd, 1))


def draw(rng: random.Random):
    path = rng.choice(["fbp", "fbp", "fbp", "fdk", "fdk", "fdk", "dd", "sf", "net", "grad"])
    if path == "fdk":
        ns, nx = _log(rng, 64, 512), _log(rng, 48, 400)
        return dict(path=path, kind=rng.choice(["flat", "flat", "arc"]), ns=ns, nt=_log(rng, 32, 384),
                    na=_views(rng, 60, 720), nx=nx, ny=nx if rng.random() < 0.5 else _log(rng, 48, 400),
                    nz=_log(rng, 24, 256), ds=1.0, dx=0.0, orbit=rng.choice([360.0, 360.0, 360.0, 0.0]),
                    offset=rng.choice([0.0, 0.25]), window=rng.choice(["none", "hann"]),
                    storage=rng.choice(["f32", "f32", "f16"]), **_scanner(rng, ns))
    if path == "grad":
        return dict(path=path, rows=_log(rng, 64, 4096), nb=_log(rng, 128, 1024))
    nb, nx = _log(rng, 64, 1024), _log(rng, 48, 640)
    kind = rng.choice(["flat", "arc"])
    if path == "dd":
        return dict(path=path, kind=kind, nb=nb, na=_views(rng, 30, 360), nx=min(nx, 512), d=1.0, dx=0.0,
                    **_scanner(rng, nb))
    ny = nx if rng.random() < 0.5 else _log(rng, 48, 640)
    if path == "sf":
        return dict(path=path, kind=rng.choice([kind, "par"]), nb=nb, na=_views(rng, 30, 360), nx=nx, ny=ny, d=1.0,
                    dx=0.0, orbit=360.0, offset=rng.choice([0.0, 0.25]), **_scanner(rng, nb))
    if path == "net":
        return dict(path=path, kind=kind, nb=nb, na=_views(rng, 45, 360), nx=nx, ny=ny, d=1.0, dx=0.0, orbit=360.0,
                    offset=0.0, window="none", slices=1, **_scanner(rng, nb))
    kind = rng.choice(["par", "arc", "flat"])
    orbit = rng.choice([180.0, 360.0]) if kind == "par" else rng.choice([360.0, 360.0, 0.0])
    return dict(path=path, kind=kind, nb=nb, na=_views(rng, 60, 1200), nx=nx, ny=ny, d=1.0, dx=0.0, orbit=orbit,
                offset=rng.choice([0.0, 0.25, 1.25]), window=rng.choice(["none", "hann"]),
                slices=rng.choice([1, 1, 1, _log(rng, 2, 16)]), **_scanner(rng, nb))


# ------------------------------------------------------------------------------- geometry

def _reach(c, n, d):
    """The detector's larger side, from the central ray."""
    return d * ((n - 1) / 2 + abs(c["offset"]))


def _orbit(c, n, d):
    """The case's orbit in degrees; 0 stands for the short scan, 180 plus the full fan."""
    if c["orbit"]:
        return c["orbit"]
    s = _reach(c, n, d)
    return 180 + 2 * math.degrees(s / c["dsd"] if c["kind"] == "arc" else math.atan(s / c["dsd"]))


def _fov(c, n, d):
    s = _reach(c, n, d)
    if c["kind"] == "par":
        return s
    return (c["dsd"] - c["dod"]) * math.sin(s / c["dsd"] if c["kind"] == "arc" else math.atan(s / c["dsd"]))


def _geom2(c):
    """(ray geometry, image geometry) of a 2D case, the image masked to the field of view."""
    kw = dict(nb=c["nb"], na=c["na"], d=c["d"], orbit=_orbit(c, c["nb"], c["d"]), offset=c["offset"])
    if c["kind"] == "par":
        rg = S.SinoPar(**kw)
    else:
        rg = (S.SinoFanArc if c["kind"] == "arc" else S.SinoFanFlat)(dsd=c["dsd"], dod=c["dod"], **kw)
    # the smaller side of the detector bounds what every view sees
    r = _fov(c, c["nb"], c["d"]) - 2 * (abs(c["offset"]) + 1) * c["d"]
    dx = c["dx"] or 1.96 * r / math.hypot(c["nx"], c["ny"])
    ig = S.ImageGeom((c["nx"], c["ny"]), (dx, dx))
    return rg, ig.with_mask(ig.circle(r))


def _geom3(c):
    cls = S.CtFanArc if c["kind"] == "arc" else S.CtFanFlat
    rg = cls(ns=c["ns"], nt=c["nt"], ds=c["ds"], dt=c["ds"], na=c["na"], orbit=_orbit(c, c["ns"], c["ds"]),
             offset_s=c["offset"], dsd=c["dsd"], dod=c["dod"])
    r = _fov(c, c["ns"], c["ds"]) - 2 * (abs(c["offset"]) + 1) * c["ds"]
    if c["dx"]:
        return rg, S.ImageGeom((c["nx"], c["ny"], c["nz"]), (c["dx"],) * 3)
    dx = 1.96 * r / math.hypot(c["nx"], c["ny"])
    zmax = 0.5 * (c["nt"] - 4) * c["ds"] * (1 - c["dod"] / c["dsd"] - r / c["dsd"])  # seen from every side
    return rg, S.ImageGeom((c["nx"], c["ny"], c["nz"]), (dx, dx, 2 * zmax / c["nz"]))


def _angles(rg):
    a = rg.orbit_start + np.arange(rg.na) * (rg.orbit / rg.na)
    return torch.as_tensor(a * (math.pi / 180), device="cuda")


def _bins(n, d, offset):
    return d * (torch.arange(n, device="cuda", dtype=torch.float64) - ((n - 1) / 2 + float(np.float32(offset))))


def _axes(ig):
    return [torch.as_tensor(a, device="cuda") for a in ig.axes()]


# --------------------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _ellipses(g, n, r, lo=0.02, hi=0.5):
    """(n, 6): centres within 0.8 r, semi-axes lo r to hi r, any angle, densities -0.3 to 1."""
    u = torch.rand(n, 6, device="cuda", generator=g, dtype=torch.float64)
    c, t = 0.8 * r * u[:, 0].sqrt(), 2 * math.pi * u[:, 1]
    return torch.stack([c * t.cos(), c * t.sin(), r * (lo + (hi - lo) * u[:, 2]), r * (lo + (hi - lo) * u[:, 3]),
                        math.pi * u[:, 4], -0.3 + 1.3 * u[:, 5]], 1)


def _ellipse_sino(rg, ell):
    """Line integrals of ellipses, (na, nb) float64."""
    s, beta = _bins(rg.nb, rg.d, rg.offset)[None, :], _angles(rg)[:, None]
    if rg.kind == "par":
        r, phi = s, beta
    else:
        gam = s / rg.dsd if rg.kind == "arc" else torch.atan(s / rg.dsd)
        r, phi = (rg.dsd - rg.dod) * gam.sin(), beta + gam
    r, phi = torch.broadcast_tensors(r, phi)
    out = torch.zeros_like(r)
    for cx, cy, rx, ry, th, rho in ell.tolist():
        rr = r - (cx * phi.cos() + cy * phi.sin())
        a2 = (rx * (phi - th).cos()) ** 2 + (ry * (phi - th).sin()) ** 2
        out += rho * 2 * rx * ry * (a2 - rr * rr).clamp_min(0).sqrt() / a2
    return out


def _noisy(x, g, sigma):
    """Detector noise of sigma times the largest line integral."""
    return x + sigma * x.abs().amax() * torch.randn(x.shape, device="cuda", generator=g, dtype=x.dtype)


def _sino(c, rg, seed):
    """A stack of noisy sinograms (slices, na, nb), or one (na, nb), float32: 0.1% of the maximum at full
    dose, and the 0.5% that the learned filter is trained for."""
    g = _gen(seed)
    sigma = 0.005 if c["path"] == "net" else 0.001
    r = 0.9 * _fov(c, c["nb"], c["d"])
    n = c.get("slices", 1)
    x = torch.stack([_noisy(_ellipse_sino(rg, _ellipses(g, 20, r)), g, sigma) for _ in range(n)]).float()
    return x if n > 1 else x[0].contiguous()


def _ellipsoid_proj(rg, ig, seed):
    """Cone-beam projections of 30 random ellipsoids inside the volume, (na, nt, ns) float32."""
    g = _gen(seed)
    x, y, z = (float(a.abs().max()) for a in _axes(ig))
    u = torch.rand(30, 8, device="cuda", generator=g)
    c = torch.stack([0.8 * x * (2 * u[:, 0] - 1), 0.8 * y * (2 * u[:, 1] - 1), 0.8 * z * (2 * u[:, 2] - 1)], 1)
    axes = torch.stack([x * (0.02 + 0.4 * u[:, 3]), y * (0.02 + 0.4 * u[:, 4]), z * (0.05 + 0.5 * u[:, 5])], 1)
    rot = torch.linalg.qr(torch.randn(30, 3, 3, device="cuda", generator=g))[0]
    A = (rot / axes[:, :, None]).double()  # the unit ball's map
    rho = (-0.3 + 1.3 * u[:, 6]).tolist()
    s, t = _bins(rg.ns, rg.ds, rg.offset_s), _bins(rg.nt, rg.dt, rg.offset_t)
    dso = rg.dsd - rg.dod
    if rg.kind == "arc":
        px, py = rg.dsd * (s / rg.dsd).sin(), dso - rg.dsd * (s / rg.dsd).cos()
    else:
        px, py = s, torch.full_like(s, dso - rg.dsd)
    out = torch.empty(rg.na, rg.nt, rg.ns, device="cuda")
    step = max(1, (1 << 26) // (rg.nt * rg.ns))
    beta = _angles(rg)
    for a in range(0, rg.na, step):
        cb, sb = beta[a:a + step].cos()[:, None, None], beta[a:a + step].sin()[:, None, None]
        src = torch.stack([-dso * sb[:, 0, 0], dso * cb[:, 0, 0], 0 * cb[:, 0, 0]], 1)
        dx = ((px * cb - py * sb) + dso * sb).float()
        dy = ((px * sb + py * cb) - dso * cb).float()
        dz = t.float()[None, :, None]
        norm2 = dx * dx + dy * dy + dz * dz
        acc = torch.zeros(norm2.shape, device="cuda")
        for e in range(30):
            M = A[e].tolist()
            q = (src - c[e].double()) @ A[e].T  # (views, 3)
            v = [m[0] * dx + m[1] * dy + m[2] * dz for m in M]
            vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2]
            uv = sum(q[:, k, None, None].float() * v[k] for k in range(3)) / vv
            # the closest approach to the centre, so that nothing cancels
            w = sum((q[:, k, None, None].float() - uv * v[k]) ** 2 for k in range(3))
            acc += (2 * rho[e]) * ((1 - w).clamp_min(0) / vv * norm2).sqrt()
        out[a:a + step] = acc
    return out


def _ellipse_image(ig, ell):
    """Pixel averages (2 x 2 samples) of ellipses, (ny, nx) float64."""
    x, y = _axes(ig)
    dx, dy = ig.deltas
    out = torch.zeros(len(y), len(x), device="cuda", dtype=torch.float64)
    for ox in (-0.25, 0.25):
        for oy in (-0.25, 0.25):
            X, Y = x[None, :] + ox * dx, y[:, None] + oy * dy
            for cx, cy, rx, ry, th, rho in ell.tolist():
                u = (X - cx) * math.cos(th) + (Y - cy) * math.sin(th)
                v = -(X - cx) * math.sin(th) + (Y - cy) * math.cos(th)
                out += (0.25 * rho) * ((u / rx) ** 2 + (v / ry) ** 2 <= 1)
    return out


def _pair_inputs(c, rg, ig, seed):
    """A solver's image (ny, nx) and, early on, its residual (na, nb): what the image still lacks, and noise."""
    g = _gen(seed)
    r = 0.9 * _fov(_pair(c), c["nb"], c["d"])
    img = _ellipse_image(ig, _ellipses(g, 20, r)).float()
    return img, _noisy(0.1 * _ellipse_sino(rg, _ellipses(g, 20, r)), g, 0.01).float()


def _net_weights():
    f = np.load(learned.default_weights_path())
    return f["params"].astype(np.float32), float(f["scale"])


def _grad_rows(c, seed):
    """Ramp-filtered detector rows with and without noise, (rows, nb) float32: a training batch."""
    rg = S.SinoFanArc(nb=c["nb"], d=1.0239 * 888 / c["nb"], na=90, orbit=360.0, dsd=949.075, dod=408.075)
    g, zn, zc = _gen(seed), [], []
    for _ in range(-(-c["rows"] // rg.na)):
        x = _ellipse_sino(rg, _ellipses(g, 20, 220.0))
        zc.append(_filter64(rg, x, "none"))
        zn.append(_filter64(rg, _noisy(x, g, 0.005), "none"))
    return [torch.cat(v)[:c["rows"]].float().contiguous() for v in (zn, zc)]


# ----------------------------------------------------------------------- prepare, run, work

def prepare(case, seed):
    c = case
    if c["path"] in ("fbp", "net"):
        rg, ig = _geom2(c)
        st = dict(c=c, plan=S.plan_fbp(rg, ig, window=S.Window(c["window"])), sino=_sino(c, rg, seed))
        if c["path"] == "net":
            p, scale = _net_weights()
            st["net"] = learned.LearnedFilter(scale, p)
        return st
    if c["path"] == "fdk":
        rg, ig = _geom3(c)
        plan = S.plan_fbp(rg, ig, window=S.Window(c["window"]), storage=c["storage"])
        return dict(c=c, plan=plan, proj=_ellipsoid_proj(rg, ig, seed))
    if c["path"] == "batch":
        rgs, igs, _ = S.random_ct_scans(c["scans"], c["geometry_seed"])
        return dict(c=c, batch=S.FDKBatch(rgs, igs, storage=c["storage"]),
                    proj=[_ellipsoid_proj(rg, ig, seed + 1000 * i) for i, (rg, ig) in enumerate(zip(rgs, igs))])
    if c["path"] == "grad":
        p, scale = _net_weights()
        z, target = _grad_rows(c, seed)
        return dict(c=c, net=learned.LearnedFilter(scale, p), z=z, target=target)
    rg, ig = _geom2(_pair(c))
    img, res = _pair_inputs(c, rg, ig, seed)
    if c["path"] == "sf":
        return dict(c=c, plan=S.SFPlan(rg, ig), img=img, res=res)
    return dict(c=c, plan=S.BddPlan(S.BddGeo.from_geoms(rg, ig)), img=learned.image_to_dd(img), res=res.T.contiguous())


def _pair(c):
    return dict(dict(orbit=360.0, offset=0.0, ny=c["nx"]), **c)


def run(state):
    path = state["c"]["path"]
    if path == "fbp":
        return S.fbp(state["plan"], state["sino"])
    if path == "net":
        return learned.fbp_learned(state["plan"], state["net"], state["sino"], judge=False)[0]
    if path == "fdk":
        return S.fdk(state["plan"], state["proj"])
    if path == "batch":
        b = state["batch"]
        for i, p in enumerate(state["proj"]):
            b.set_input(i, p)
        b.run()
        return [b.get_output(i, device=True) for i in range(len(b))]
    if path == "grad":
        loss, grads = state["net"].loss_grad(state["z"], state["target"])
        return {"loss": loss, "grads": grads}
    # an iterative solver enqueues its projections one after another and waits once
    return {"sino": state["plan"].project(state["img"], sync=False),
            "image": state["plan"].backproject(state["res"], sync=False)}


_CNN = sum(ci * co * 9 for ci, co in ((1, 32), (32, 32), (32, 32), (32, 32), (32, 1)))  # per sample


def work(case):
    c = case
    if c["path"] in ("fbp", "net"):
        n, rows = c["slices"], c["slices"] * c["na"]
        pix, net = math.pi / 4 * c["nx"] * c["ny"], _CNN if c["path"] == "net" else 0
        return {"bytes": 4 * (rows * c["nb"] + n * c["nx"] * c["ny"]),
                "flops": 12 * pix * rows + rows * _fft_flops(c["nb"]) + 2 * net * rows * c["nb"]}
    if c["path"] == "fdk":
        return _fdk_work(c["ns"], c["nt"], c["na"], c["nx"], c["ny"], c["nz"])
    if c["path"] == "batch":
        rgs, igs, _ = S.random_ct_scans(c["scans"], c["geometry_seed"])
        each = [_fdk_work(r.ns, r.nt, r.na, *i.dims) for r, i in zip(rgs, igs)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if c["path"] == "grad":
        return {"bytes": 8 * c["rows"] * c["nb"], "flops": 6 * _CNN * c["rows"] * c["nb"]}
    ny = c.get("ny", c["nx"])
    per = 10 if c["path"] == "dd" else 40  # per pixel and view, either direction
    return {"bytes": 8 * (c["nx"] * ny + c["na"] * c["nb"]), "flops": 2 * per * c["nx"] * ny * c["na"]}


def _fft_flops(n):
    npad = 1 << int(math.ceil(math.log2(n + 1)))
    return 5 * npad * math.log2(npad)


def _fdk_work(ns, nt, na, nx, ny, nz):
    return {"bytes": 4 * (ns * nt * na + nx * ny * nz), "flops": 15 * nx * ny * nz * na + nt * na * _fft_flops(ns)}


# ------------------------------------------------------------------------- exact, in 64 bits

def _filter64(rg, x, window, first=0):
    """Weighted, ramp-filtered rows of float64 data by FFT: views first, first + 1, ... of the scan in
    the leading axis (second to last for a stack of sinograms)."""
    ct = hasattr(rg, "ns")
    n, d = (rg.ns, rg.ds) if ct else (rg.nb, rg.d)
    s, beta = _bins(n, d, rg.offset_s if ct else rg.offset), _angles(rg)
    beta, start = beta[first:first + x.shape[0 if ct else -2]], beta.min()
    npad = 1 << int(math.ceil(math.log2(n + 1)))
    k = torch.arange(npad, device="cuda", dtype=torch.float64) - npad // 2
    den = math.pi * (rg.dsd * torch.sin(k * d / rg.dsd) if rg.kind == "arc" else k * d)
    h = torch.where(k % 2 != 0, -1 / den ** 2, torch.zeros_like(k))
    h[npad // 2] = 0.25 / d ** 2
    H = torch.fft.fft(torch.fft.ifftshift(h)).real * d / torch.fft.ifftshift(torch.sinc(k / npad)) ** 2
    if window == "hann":
        w = 0.5 * (1 + torch.cos(2 * math.pi * k / npad)) * (k.abs() < npad / 2)
        H = H * torch.fft.ifftshift(w.float().double())
    # view weights: angle step over the number of times each line is measured, and Parker's
    step = abs(math.radians(rg.orbit / rg.na))
    x = x * (step / max(1, math.floor(1.00001 * step * rg.na / math.pi)))
    if rg.kind != "par":
        gam = s / rg.dsd if rg.kind == "arc" else torch.atan(s / rg.dsd)
        if math.trunc(rg.orbit / 360) * 360 != rg.orbit:
            b, gm = (beta - start)[:, None], gam.abs().max()
            up = torch.sin(math.pi / 2 * b / (2 * (gm - gam))) ** 2
            down = torch.sin(math.pi / 2 * (math.pi + 2 * gm - b) / (2 * (gm + gam))) ** 2
            w = torch.where(b < 2 * (gm - gam), up, torch.zeros_like(up))
            w = torch.where((2 * (gm - gam) <= b) & (b < math.pi - 2 * gam), torch.ones_like(w), w)
            w = torch.where((math.pi - 2 * gam < b) & (b <= math.pi + 2 * gm), down, w)
            x = x * (w[:, None, :] if ct else w)
        dso = rg.dsd - rg.dod
        if not ct:
            x = x * (dso * gam.cos()).abs() / rg.dsd
        else:
            t = _bins(rg.nt, rg.dt, rg.offset_t)[:, None]
            if rg.kind == "arc":
                x = x * ((dso / rg.dsd) * gam.cos() / torch.sqrt((t / rg.dsd) ** 2 + 1))
            else:
                x = x * (dso / torch.sqrt(s ** 2 + t ** 2 + rg.dsd ** 2))
    elif math.trunc(rg.orbit / 180) * 180 != rg.orbit:
        raise ValueError("parallel beams take whole half turns here")
    return torch.fft.irfft(torch.fft.rfft(x, npad) * H[:npad // 2 + 1], npad)[..., :n]


def _column64(rg, n, d, offset, X, Y, b):
    """Detector position (1-based), magnification and weight of the points (X, Y) in view angle b."""
    w = (n + 1) / 2 + float(np.float32(offset))
    xb, yb = (X * math.cos(b) + Y * math.sin(b)) / d, (-X * math.sin(b) + Y * math.cos(b)) / d
    if rg.kind == "par":
        return xb + w, None, None
    dsd, yb = rg.dsd / d, (rg.dsd - rg.dod) / d - yb
    if rg.kind == "arc":
        return dsd * torch.atan2(xb, yb) + w, dsd / yb, dsd ** 2 / (xb * xb + yb * yb)
    return dsd / yb * xb + w, dsd / yb, (dsd / yb) ** 2


def _back64(rg, ig, rows):
    """Pixel-driven back-projection of filtered rows (slices, na, nb): (slices, ny, nx)."""
    x, y = _axes(ig)
    keep = torch.as_tensor(ig.mask, device="cuda")
    Y, X = (v[keep] for v in torch.meshgrid(y, x, indexing="ij"))
    acc = torch.zeros(rows.shape[0], X.numel(), device="cuda", dtype=torch.float64)
    for v, b in enumerate(_angles(rg).tolist()):
        bb, _, w2 = _column64(rg, rg.nb, rg.d, rg.offset, X, Y, b)
        i = bb.floor()
        ok = (i >= 1) & (i < rg.nb)
        f, i = bb - i, i.clamp(1, rg.nb - 1).long()
        r = rows[:, v]
        acc += ((1 - f) * r[:, i - 1] + f * r[:, i]) * (ok if w2 is None else ok * w2)
    out = torch.zeros(rows.shape[0], len(y), len(x), device="cuda", dtype=torch.float64)
    out[:, keep] = acc
    return out


def _fdk64(rg, ig, proj, window):
    x, y, z = _axes(ig)
    Y, X = (v.reshape(-1) for v in torch.meshgrid(y, x, indexing="ij"))
    out = torch.zeros(len(z), X.numel(), device="cuda", dtype=torch.float64)
    wt = (rg.nt + 1) / 2 + float(np.float32(rg.offset_t))
    q = torch.cat([_filter64(rg, p.double(), window, 32 * i) for i, p in enumerate(proj.split(32))])
    for v, b in enumerate(_angles(rg).tolist()):
        bs, mag, w2 = _column64(rg, rg.ns, rg.ds, rg.offset_s, X, Y, b)
        i = bs.floor()
        ok = (i >= 1) & (i < rg.ns)
        f, i = bs - i, i.clamp(1, rg.ns - 1).long()
        prof = q[v].T.contiguous()  # (ns, nt)
        prof = (w2 * ok)[:, None] * torch.lerp(prof[i - 1], prof[i], f[:, None])  # (columns, nt)
        bt = mag[:, None] * (z / rg.dt)[None] + wt
        it = bt.floor()
        bt -= it
        valid = (it >= 1) & (it < rg.nt)
        it = it.clamp_(1, rg.nt - 1).long()
        val = torch.lerp(prof.gather(1, it - 1), prof.gather(1, it), bt)
        out += (val * valid).T
    return out.reshape(len(z), len(y), len(x))


def _net64(z, params, scale):
    """z + scale * net(z / scale) on rows (R, L); weights rounded to bfloat16 as the network defines them."""
    h, o = (z / scale)[:, None], 0
    for k, (ci, co) in enumerate(((1, 32), (32, 32), (32, 32), (32, 32), (32, 1))):
        w = params[o:o + 9 * ci * co].reshape(co, ci, 9)
        b = params[o + 9 * ci * co:o + 9 * ci * co + co]
        o += 9 * ci * co + co
        w = w + (w.detach().float().bfloat16().double() - w.detach())
        h = torch.einsum("ock,rclk->rol", w, torch.nn.functional.pad(h, (4, 4)).unfold(2, 9, 1)) + b[None, :, None]
        if k < 4:
            h = torch.nn.functional.gelu(h)
    return z + scale * h[:, 0]


def _dd64(geo, img, res):
    """The branchless distance-driven pair: sinogram (nDet, na) of img, image of res (nDet, na)."""
    n, nd, p = geo.nPix, geo.nDet, geo.pSize
    f64 = dict(device="cuda", dtype=torch.float64)
    k = torch.arange(nd + 1, **f64) - nd / 2
    if geo.arc:
        ux, uy = geo.DSD * torch.sin(k * geo.dSize / geo.DSD), geo.DS0 - geo.DSD * torch.cos(k * geo.dSize / geo.DSD)
    else:
        ux, uy = k * geo.dSize, torch.full_like(k, -(geo.DSD - geo.DS0) - geo.dSize / 2)
    r, c = torch.arange(n, **f64)[:, None], torch.arange(n + 1, **f64)[None, :]
    sino, image = torch.zeros(nd, len(geo.angle), **f64), torch.zeros(n, n, **f64)

    def interp(kn, v, q):  # piecewise linear along the last axis, held at the ends
        kn, v, q = (torch.broadcast_to(w, (n, w.shape[-1])).contiguous() for w in (kn, v, q))
        j = torch.searchsorted(kn, q, right=True).clamp(1, kn.shape[1] - 1)
        a, b = kn.gather(1, j - 1), kn.gather(1, j)
        t = ((q - a) / (b - a)).clamp(0, 1)
        return torch.lerp(v.gather(1, j - 1), v.gather(1, j), t)

    for v, b in enumerate(geo.angle.tolist()):
        tx, ty = -geo.DS0 * math.sin(b), geo.DS0 * math.cos(b)
        rx, ry = ux * math.cos(b) - uy * math.sin(b), ux * math.sin(b) + uy * math.cos(b)
        rows = not (math.pi / 4 <= b <= 3 * math.pi / 4 or 5 * math.pi / 4 <= b <= 7 * math.pi / 4)
        if rows:  # onto the x axis, image rows
            det = tx - ty * (tx - rx) / (ty - ry)
            X, Yc = (c - n / 2) * p, (n / 2 - 0.5 - r) * p
            edge = tx - ty * (tx - X) / (ty - Yc)
            cos = torch.cos(torch.atan((tx - (det[1:] + det[:-1]) / 2).abs() / abs(ty)))
            val = img.T
        else:  # onto the y axis, image columns
            det = ty - tx * (ty - ry) / (tx - rx)
            X, Yc = (r - n / 2) * p, (c - n / 2 - 0.5) * p
            edge = ty - tx * (ty - Yc) / (tx - X)
            cos = torch.sin(torch.atan(abs(tx) / (ty - (det[1:] + det[:-1]) / 2).abs()))
            val = img.flip(1)
        L = (p / ((det[1:] - det[:-1]) * cos)).abs()
        P = torch.nn.functional.pad((val * edge.diff(dim=1)).cumsum(1), (1, 0))
        sino[:, v] = interp(edge, P, det[None]).diff(dim=1).abs().sum(0) * L
        Q = torch.nn.functional.pad((res[:, v] * L * det.diff()).cumsum(0), (1, 0))
        kn, Q = (det.flip(0), Q.flip(0)) if det[0] > det[1] else (det, Q)
        add = interp(kn[None], Q[None], edge).diff(dim=1).abs()
        image += add.T if rows else add.flip(1)
        if v == 0:  # the reference's first view counts twice, in this layout
            image += add.T
    return sino, image


def _sf64(rg, ig, img, res):
    """The separable-footprint pair (trapezoid footprints, chord amplitude): sinogram and image."""
    x, y = _axes(ig)
    keep = torch.as_tensor(ig.mask, device="cuda")
    Y, X = (v[keep] for v in torch.meshgrid(y, x, indexing="ij"))
    hx, hy = abs(ig.deltas[0]) / 2, abs(ig.deltas[1]) / 2
    val, acc = img[keep], torch.zeros_like(X)
    sino = torch.zeros(rg.na, rg.nb, device="cuda", dtype=torch.float64)
    for v, b in enumerate(_angles(rg).tolist()):
        corners = [(X + i * hx, Y + j * hy) for i in (-1, 1) for j in (-1, 1)]
        t = torch.stack([_column64(rg, rg.nb, rg.d, rg.offset, *xy, b)[0] - 1 for xy in corners]).sort(0)[0]
        if rg.kind == "par":
            ex, ey = torch.full_like(X, -math.sin(b)), torch.full_like(X, math.cos(b))
        else:
            dso = rg.dsd - rg.dod
            ex, ey = X + dso * math.sin(b), Y - dso * math.cos(b)
            ex, ey = ex / torch.hypot(ex, ey), ey / torch.hypot(ex, ey)
        h = 4 * hx * hy / torch.maximum(2 * hy * ex.abs(), 2 * hx * ey.abs())

        def cdf(u):
            a, m, z = u.clamp(min=t[0], max=t[1]), u.clamp(min=t[1], max=t[2]), u.clamp(min=t[2], max=t[3])
            up = torch.where(t[1] > t[0], (a - t[0]) ** 2 / (2 * (t[1] - t[0])), torch.zeros_like(a))
            dn = torch.where(t[3] > t[2], ((t[3] - t[2]) ** 2 - (t[3] - z) ** 2) / (2 * (t[3] - t[2])), torch.zeros_like(z))
            return up + (m - t[1]) + dn

        k0 = torch.ceil(t[0] - 0.5)
        last = cdf(k0 - 0.5)
        for k in range(int((t[3] - t[0]).max()) + 3):
            nxt = cdf(k0 + k + 0.5)
            g, last = h * (nxt - last), nxt
            ok = (k0 + k >= 0) & (k0 + k < rg.nb)
            i = (k0 + k).clamp(0, rg.nb - 1).long()
            g = g * ok
            sino[v].index_add_(0, i, g * val)
            acc += g * res[v][i]
    out = torch.zeros(len(y), len(x), device="cuda", dtype=torch.float64)
    out[keep] = acc
    return sino, out


def exact(case, seed):
    c = case
    if c["path"] in ("fbp", "net"):
        rg, ig = _geom2(c)
        sino = _sino(c, rg, seed).double()
        rows = _filter64(rg, sino.reshape(-1, rg.na, rg.nb), c["window"])
        if c["path"] == "net":
            p, scale = _net_weights()
            p = torch.as_tensor(p, device="cuda").double()
            rows = torch.cat([_net64(r, p, scale) for r in rows.reshape(-1, rg.nb).split(128)]).reshape(rows.shape)
        return _back64(rg, ig, rows).reshape(tuple(sino.shape[:-2]) + (c["ny"], c["nx"]))
    if c["path"] == "fdk":
        rg, ig = _geom3(c)
        return _fdk64(rg, ig, _ellipsoid_proj(rg, ig, seed), c["window"])
    if c["path"] == "batch":
        rgs, igs, _ = S.random_ct_scans(c["scans"], c["geometry_seed"])
        return [_fdk64(rg, ig, _ellipsoid_proj(rg, ig, seed + 1000 * i), "none") for i, (rg, ig) in enumerate(zip(rgs, igs))]
    if c["path"] == "grad":
        p, scale = _net_weights()
        p = torch.as_tensor(p, device="cuda").double().requires_grad_()
        z, t = _grad_rows(c, seed)
        loss = 0.0
        for a, b in zip(z.split(64), t.split(64)):
            part = ((_net64(a.double(), p, scale) - b) ** 2).sum() / (scale ** 2 * z.numel())
            part.backward()
            loss += float(part)
        return {"loss": loss, "grads": p.grad.cpu().numpy()}
    rg, ig = _geom2(_pair(c))
    img, res = (v.double() for v in _pair_inputs(c, rg, ig, seed))
    if c["path"] == "sf":
        sino, image = _sf64(rg, ig, img, res)
    else:
        sino, image = _dd64(S.BddGeo.from_geoms(rg, ig), learned.image_to_dd(img), res.T)
    return {"sino": sino, "image": image}
