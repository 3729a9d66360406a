"""Performance cases of the strip and 3D hybrid list-mode TOF MLEM.

Each case is work that a program using ``stripmlem`` has it do, through the
package's public entry points:

* ``new``      new list-mode events into a context, a few MLEM iterations from
               a uniform image, the image back (the whole life of one
               reconstruction);
* ``mlem``     MLEM / OSEM iterations over resident events from a uniform
               image, in either mode, and the image back;
* ``batch``    several reconstructions advanced together;
* ``project``  the differentiable projection: forward, and backward to the
               image and, where asked for, to the two sigmas;
* ``hybrid``   the 3D hybrid reconstruction: resident responses, or new ones
               in every pass, MLEM iterations, the volume back.

``exact`` restates the mathematics in 64 bits with plain torch: the pixel
sets and the frame events are decided in binary32 as the model defines them,
the rest is binary64.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "j-pet-mlem-old_b200"))

import stripmlem as sm  # noqa: E402
from stripmlem import autograd as sag  # noqa: E402
from stripmlem import hybrid as hy  # noqa: E402

DEV = "cuda:0"
NOISE_SEED = 7919
# exact() leaves a case out when it has more kernel evaluations than this
EXACT_MOST = 2.5e10

# Strip geometries: radius, length, rows, columns, pixel, sigma_z, sigma_dl (mm)
SMALL = (200.0, 500.0, 200, 250, 2.0, 10.0, 42.0)
LARGE = (400.0, 800.0, 400, 800, 1.0, 5.0, 25.0)
SQUARE = (200.0, 400.0, 400, 400, 1.0, 8.0, 30.0)
WIDE = (150.0, 437.0, 300, 437, 1.0, 10.0, 42.0)


def _strip(kind, geometry, events, **more):
    R, L, n_y, n_z, p, s_z, s_dl = geometry
    return dict(kind=kind, radius=R, length=L, n_y=n_y, n_z=n_z, pixel=p, s_z=s_z, s_dl=s_dl,
                events=events, **more)


def _hybrid(n_pix, responses, iterations, resident):
    return dict(kind="hybrid", n_pix=n_pix, responses=responses, iterations=iterations,
                resident=resident)


def listed():
    return [
        # a quick look at a short run: 20 000 events just taken, five
        # iterations on the small scanner (launches and host time count)
        dict(name="new_small", **_strip("new", SMALL, 20_000, iterations=5, accum="kahan")),
        # an ordinary acquisition read into host memory and reconstructed at
        # the fine resolution, events and all
        dict(name="new_large", **_strip("new", LARGE, 5_000_011, iterations=10, accum="kahan")),
        # iterating on resident events, coarse pixels, binary64 row sums
        dict(name="mlem_small", **_strip("mlem", SMALL, 1_000_003, iterations=5, subsets=1,
                                         mode="cpu", accum="fp64")),
        # the long acquisition at the fine resolution: iterations over 1e8 events
        dict(name="mlem_large", **_strip("mlem", LARGE, 100_000_000, iterations=2, subsets=1,
                                         mode="cpu", accum="kahan")),
        # ordered subsets over a medium event list
        dict(name="osem8_large", **_strip("mlem", LARGE, 8_000_009, iterations=2, subsets=8,
                                          mode="cpu", accum="kahan")),
        # broad TOF resolution on fine pixels: the tallest event boxes
        dict(name="mlem_wide", **_strip("mlem", WIDE, 2_000_003, iterations=3, subsets=1,
                                        mode="cpu", accum="kahan")),
        # the sensitivity-normalised update with the analytic kernel
        dict(name="analytic_small", **_strip("mlem", SMALL, 500_009, iterations=3, subsets=1,
                                             mode="gpu", accum="kahan")),
        # a slice stack: eight reconstructions of mixed size together
        dict(name="batch8", kind="batch", members=8, first=3, scale=0.25, iterations=3),
        # list-mode likelihood step of a learned model: projection of the
        # image and its gradient
        dict(name="project_large", **_strip("project", LARGE, 20_000_003, sigma=False)),
        # the same with the gradient to the resolution parameters (sigma fit)
        dict(name="project_sigma", **_strip("project", SQUARE, 2_000_003, sigma=True)),
        # 3D hybrid, coarse voxels, a short list of new responses per pass
        dict(name="hybrid_small", **_hybrid(50, 50_000, 3, False)),
        # 3D hybrid at the big barrel's full grid
        dict(name="hybrid_large", **_hybrid(200, 10_000_000, 4, True)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: fields of 100-800 pixels of 1-4 mm,
    sigmas 5-10 and 25-42 mm, 1e4 to 2e7 events; hybrid grids of 40-120
    pixels and 1e4 to 2e6 responses."""
    kind = rng.choice(["new", "mlem", "mlem", "osem", "analytic", "project", "sigma", "batch",
                       "hybrid", "hybrid"])
    if kind == "hybrid":
        return _hybrid(rng.randint(40, 120), _log_int(rng, 10_000, 2_000_000), rng.randint(1, 4),
                       rng.random() < 0.5)
    if kind == "batch":
        return dict(kind="batch", members=rng.randint(2, 12), first=rng.randint(0, 1000),
                    scale=math.exp(rng.uniform(math.log(0.05), math.log(0.3))),
                    iterations=rng.randint(1, 4))
    n_y, n_z, p = rng.randint(100, 500), rng.randint(100, 800), float(rng.randint(1, 4))
    g = (n_y * p / 2.0, n_z * p, n_y, n_z, p, round(rng.uniform(5.0, 10.0), 2),
         round(rng.uniform(25.0, 42.0), 2))
    accum = rng.choice(["kahan", "kahan", "fp32", "fp64"])
    if kind == "new":
        return _strip("new", g, _log_int(rng, 10_000, 5_000_000), iterations=rng.randint(2, 10),
                      accum=accum)
    if kind == "mlem":
        return _strip("mlem", g, _log_int(rng, 20_000, 20_000_000), iterations=rng.randint(1, 5),
                      subsets=1, mode="cpu", accum=accum)
    if kind == "osem":
        return _strip("mlem", g, _log_int(rng, 100_000, 10_000_000), iterations=rng.randint(1, 3),
                      subsets=rng.choice([2, 4, 8, 16]), mode="cpu", accum=accum)
    if kind == "analytic":
        return _strip("mlem", g, _log_int(rng, 20_000, 2_000_000), iterations=rng.randint(1, 3),
                      subsets=1, mode="gpu", accum=accum)
    if kind == "project":
        return _strip("project", g, _log_int(rng, 20_000, 20_000_000), sigma=False)
    return _strip("project", g, _log_int(rng, 20_000, 2_000_000), sigma=True)


# ---- inputs ------------------------------------------------------------------

def _phantom(R, L, seed):
    """Hot and cold ellipses in a body (z, y, a, b, activity), first on top."""
    r = np.random.default_rng(seed)
    k = int(r.integers(3, 10))
    out = [(r.uniform(-0.3, 0.3) * L, r.uniform(-0.3, 0.3) * R, r.uniform(0.04, 0.15) * L,
            r.uniform(0.04, 0.15) * R, r.uniform(0.1, 2.0)) for _ in range(k)]
    return out + [(0.0, 0.0, 0.42 * L, 0.42 * R, 1.0)]


def _events(R, L, s_z, s_dl, n, seed):
    """Detected, smeared events (z_u, z_d, dl) of the phantom, on the GPU."""
    ph = _phantom(R, L, seed)
    g = torch.Generator(device=DEV).manual_seed(NOISE_SEED + seed)
    zb, yb, ab, bb, _ = ph[-1]
    out, got = [], 0
    f32 = torch.float32

    def uniform(m):
        return torch.rand(m, generator=g, device=DEV, dtype=f32)

    top = max(p[4] for p in ph)
    while got < n:
        m = int((n - got) * 3) + 4096
        m = min(m, 40_000_000)
        r, a = torch.sqrt(uniform(m)), uniform(m) * (2 * math.pi)
        z, y = zb + ab * r * torch.cos(a), yb + bb * r * torch.sin(a)
        act = torch.full_like(z, ph[-1][4])
        for cz, cy, ea, eb, v in reversed(ph[:-1]):
            act = torch.where(((z - cz) / ea) ** 2 + ((y - cy) / eb) ** 2 <= 1.0,
                              torch.full_like(act, v), act)
        t = (uniform(m) - 0.5) * (L / R)
        zu, zd = z + (R - y) * t, z - (R + y) * t
        ok = (uniform(m) * top < act) & (zu.abs() < L / 2) & (zd.abs() < L / 2)
        zu, zd, y, t = zu[ok], zd[ok], y[ok], t[ok]
        k = min(n - got, zu.numel())
        noise = torch.randn(3, zu.numel(), generator=g, device=DEV, dtype=f32)
        dl = -2.0 * y * torch.sqrt(1.0 + t * t)
        out.append((zu[:k] + s_z * noise[0, :k], zd[:k] + s_z * noise[1, :k],
                    dl[:k] + s_dl * noise[2, :k]))
        got += k
    return tuple(torch.cat([o[i] for o in out]).contiguous() for i in range(3))


def _scanner(c):
    return sm.Scanner(c["radius"], c["length"], c["n_y"], c["n_z"], c["pixel"], c["pixel"],
                      c["s_z"], c["s_dl"])


ACCUM = {"kahan": sm.ACCUM_KAHAN, "fp32": sm.ACCUM_FP32, "fp64": sm.ACCUM_FP64}


def _case_events(c, seed):
    return _events(c["radius"], c["length"], c["s_z"], c["s_dl"], c["events"], seed)


def _members(c):
    """The batch's reconstructions: fields and event counts as mixed as a
    slice stack's, sigma_z 10 mm, sigma_dl 42 mm."""
    out = []
    for i in range(c["members"]):
        r = np.random.default_rng(c["first"] + i)
        n_y, n_z = (int(v) for v in r.integers(100, 500, size=2))
        p = float(r.integers(1, 5))
        n = int(c["scale"] * math.exp(r.uniform(math.log(1e5), math.log(4e6))))
        out.append(_strip("mlem", (n_y * p / 2.0, n_z * p, n_y, n_z, p, 10.0, 42.0), n,
                          iterations=c["iterations"], subsets=1, mode="cpu", accum="kahan"))
    return out


def _project_inputs(c, seed):
    """An activity image, as a model would hold it, and the loss's gradient
    weights (positive, spread over a factor of a few)."""
    g = torch.Generator(device=DEV).manual_seed(NOISE_SEED + 31 * seed)
    rho = torch.exp(0.5 * torch.randn(c["n_y"], c["n_z"], generator=g, device=DEV))
    w = torch.exp(0.4 * torch.randn(c["events"], generator=g, device=DEV))
    return rho, w


def prepare(case, seed):
    c = case
    if c["kind"] == "hybrid":
        return _prepare_hybrid(c, seed)
    if c["kind"] == "batch":
        recs = []
        for i, m in enumerate(_members(c)):
            rec = sm.Reconstruction(_scanner(m))
            rec.set_events_device(*_settled(_case_events(m, seed + 101 * i)))
            recs.append(rec)
        return dict(case=c, recs=recs, ones=[_ones(m) for m in _members(c)],
                    batch=sm.Batch(recs))
    sc = _scanner(c)
    mode = sm.MODE_GPU if c.get("mode") == "gpu" else sm.MODE_CPU
    rec = sm.Reconstruction(sc, mode=mode, accumulation=ACCUM[c.get("accum", "kahan")])
    ev = _settled(_case_events(c, seed))
    s = dict(case=c, rec=rec, ones=_ones(c))
    if c["kind"] == "new":
        s["events"] = tuple(e.cpu().numpy() for e in ev)
    else:
        rec.set_events_device(*ev, n_subsets=c.get("subsets", 1))
    if c["kind"] == "project":
        s["rho"], s["w"] = _project_inputs(c, seed)
        s["sigma"] = torch.tensor([0.9 * c["s_z"], 0.95 * c["s_dl"]] if c["sigma"]
                                  else [c["s_z"], c["s_dl"]], dtype=torch.float32)
        s["rho"].requires_grad_(True)
        s["sigma"].requires_grad_(c["sigma"])
    return s


def _settled(t):
    torch.cuda.synchronize()  # the context works on a stream of its own
    return t


def _ones(c):
    return np.ones((c["n_y"], c["n_z"]), np.float32)


def run(state):
    s = state
    c = s["case"]
    if c["kind"] == "new":
        rec = s["rec"]
        rec.set_events(*s["events"])
        rec.rho = s["ones"]
        rec(None, c["iterations"])
        return rec.rho
    if c["kind"] == "mlem":
        rec = s["rec"]
        rec.rho = s["ones"]
        rec(None, c["iterations"])
        return rec.rho
    if c["kind"] == "batch":
        for rec, ones in zip(s["recs"], s["ones"]):
            rec.rho = ones
        s["batch"](c["iterations"])
        return [rec.rho for rec in s["recs"]]
    if c["kind"] == "project":
        # the model around the projection is binary32, like the image
        y = sag.project(s["rec"], s["rho"], s["sigma"]).to(torch.float32)
        wrt = [s["rho"], s["sigma"]] if c["sigma"] else [s["rho"]]
        return [y.detach(), *torch.autograd.grad(y, wrt, s["w"])]
    rec = s["rec"]
    if not c["resident"]:
        rec.set_responses(*s["responses"])
    rec.rho = s["ones"]
    rec(c["iterations"])
    return rec.rho


# ---- the 3D hybrid scanner -------------------------------------------------------

LENGTH, H_SIGMA_Z, H_SIGMA_DL, FOV, N_EMISSIONS = 0.5, 0.015, 0.06, 0.4, 100000
CYLINDERS = [(0.1, 0.05, 0.02, 0.05, 0.05, 3.0), (-0.15, 0.0, -0.05, 0.04, 0.08, 0.2),
             (0.0, 0.0, 0.0, 0.3, 0.2, 1.0)]


def _grid(n_pix):
    """Pixel size, planes and left end of a grid over the field of view."""
    p = 2 * FOV / n_pix
    planes = int(LENGTH / p + 1e-9)
    return p, planes, -planes * p / 2


@functools.lru_cache(maxsize=2)
def _barrel_geometry(n_pix):
    """The big barrel (three rings of 48, 48 and 96 square detectors) and its
    flattened geometry: per LOR the pixels within its detectors' width, their
    positions along it and weights falling off with the distance."""
    barrel = hy.Barrel()
    p, _, _ = _grid(n_pix)
    f64 = dict(device=DEV, dtype=torch.float64)
    cen = torch.from_numpy(barrel.centers.astype(np.float64)).to(DEV)
    poly = torch.from_numpy(barrel.polygons.astype(np.float64)).to(DEV)
    nd = barrel.n_detectors
    ax = -FOV + (torch.arange(n_pix, **f64) + 0.5) * p
    iy, ix = torch.meshgrid(torch.arange(n_pix, device=DEV), torch.arange(n_pix, device=DEV),
                            indexing="ij")
    inside = ax[ix] ** 2 + ax[iy] ** 2 <= FOV * FOV
    ix, iy = ix[inside], iy[inside]
    cx, cy = ax[ix], ax[iy]
    a_all, b_all = (torch.from_numpy(v).to(DEV) for v in np.tril_indices(nd))
    n_lors = len(a_all)
    seg = torch.cat([cen[b_all], cen[a_all]], 1)
    lor, pix, pos, hits = [], [], [], []
    for s0 in range(0, n_lors, 512):
        a, b = a_all[s0:s0 + 512], b_all[s0:s0 + 512]
        st, v = cen[b], cen[a] - cen[b]
        ln = torch.hypot(v[:, 0], v[:, 1]).clamp_min(1e-30)
        d = v / ln[:, None]
        nrm = torch.stack([-d[:, 1], d[:, 0]], 1)
        off = (st * nrm).sum(1)
        half = sum(((poly[q] * nrm[:, None, :]).sum(2) - off[:, None]).abs().amax(1)
                   for q in (a, b)) / 2 + p / 2
        dist = (cx[None] * nrm[:, :1] + cy[None] * nrm[:, 1:] - off[:, None]).abs()
        t = ((cx[None] - st[:, :1]) * d[:, :1] + (cy[None] - st[:, 1:]) * d[:, 1:]) / ln[:, None]
        li, k = torch.nonzero((dist < half[:, None]) & (t > 0) & (t < 1) & (a != b)[:, None],
                              as_tuple=True)
        lor.append(li + s0)
        pix.append(torch.stack([ix[k], iy[k]], 1))
        pos.append(t[li, k].to(torch.float32))
        hits.append(1 + torch.floor(999 * (1 - dist[li, k] / half[li])))
    lor, pix, pos, hits = (torch.cat(v) for v in (lor, pix, pos, hits))
    order = torch.sort(lor * 4.0 + pos.double(), stable=True).indices
    lor, pix, pos, hits = lor[order], pix[order], pos[order], hits[order]
    ends = torch.cumsum(torch.bincount(lor, minlength=n_lors), 0)
    begins = torch.cat([ends.new_zeros(1), ends[:-1]])
    weights = hits.to(torch.float32) / torch.tensor(float(N_EMISSIONS), device=DEV)
    host = dict(segments=seg.to(torch.float32), pixels=pix.to(torch.int16), positions=pos,
                weights=weights, lor_begin=begins, lor_end=ends)
    return barrel, {k: v.cpu().numpy() for k, v in host.items()}


def _responses(c, barrel, seed):
    return hy.generate_responses(barrel, CYLINDERS, c["responses"], LENGTH, H_SIGMA_Z, H_SIGMA_DL,
                                 seed=NOISE_SEED + seed, device=0)


def _prepare_hybrid(c, seed):
    barrel, geo = _barrel_geometry(c["n_pix"])
    p, planes, z_left = _grid(c["n_pix"])
    rec = hy.HybridReconstruction(c["n_pix"], c["n_pix"], planes, p, z_left, LENGTH, H_SIGMA_Z,
                                  H_SIGMA_DL)
    rec.set_geometry_soa(barrel.n_detectors, geo["segments"], geo["pixels"], geo["positions"],
                         geo["weights"], geo["lor_begin"], geo["lor_end"])
    rec.set_sensitivity()
    s = dict(case=c, rec=rec, ones=np.ones(rec.shape, np.float32),
             responses=_responses(c, barrel, seed))
    if c["resident"]:
        rec.set_responses(*s.pop("responses"))
    return s


# ---- work ---------------------------------------------------------------------------

def _pixels_per_event(c):
    """In-ellipse pixels: the 3-sigma ellipse's area over a pixel's, at a
    typical sec of 1.08."""
    return 9 * math.pi * c["s_z"] * c["s_dl"] / (2 * math.sqrt(2) * 1.08) / c["pixel"] ** 2


def _voxels_per_event(c):
    p = 2 * FOV / c["n_pix"]
    return (2 * 0.045 / p) * (3 * H_SIGMA_DL / 1.1 / p) * ((0.012 + p) / p)


def work(case):
    """Per kernel value and pass over it two multiplications, and a fused
    multiply-add (the projection) or an addition (the backprojection); every
    event read once per iteration, images read and written."""
    c = case
    if c["kind"] == "batch":
        parts = [work(m) for m in _members(c)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    if c["kind"] == "hybrid":
        p, planes, _ = _grid(c["n_pix"])
        it, n = c["iterations"], c["responses"]
        return {"bytes": it * (16.0 * n + 8.0 * c["n_pix"] ** 2 * planes),
                "flops": it * 8.0 * n * _voxels_per_event(c)}
    n, px = c["events"], c["n_y"] * c["n_z"]
    if c["kind"] == "project":
        return {"bytes": 2 * 12.0 * n + 8.0 * n + 8.0 * px,
                "flops": n * _pixels_per_event(c) * (8.0 + (8.0 if c["sigma"] else 0.0))}
    it = c["iterations"]
    return {"bytes": it * (12.0 * n + 8.0 * px * c.get("subsets", 1)),
            "flops": it * 8.0 * n * _pixels_per_event(c)}


# ---- 64 bits --------------------------------------------------------------------------

class _Strip64:
    """The strip model: pixel sets decided in binary32, values in binary64."""

    def __init__(self, c, events):
        f = np.float32
        self.c = c
        R, pw = f(c["radius"]), f(c["pixel"])
        n_y, n_z = c["n_y"], c["n_z"]
        sz, sdl = f(c["s_z"]), f(c["s_dl"])
        tl_y, tl_z = f(n_y) * pw / f(2), -(f(n_z) * pw) / f(2)
        ipz, ipdl = f(1) / (sz * sz), f(1) / (sdl * sdl)
        # binary32 tensors throughout: one rounding per operation
        k = lambda v: torch.tensor(float(f(v)), device=DEV, dtype=torch.float32)  # noqa: E731
        zu, zd, dl = events
        tan = (zu - zd) / k(f(2) * R)
        tt = tan * tan
        sec = torch.sqrt(k(1) + tt)
        y = k(-0.5) * (dl / sec)
        z = k(0.5) * ((zu + zd) + (k(2) * y) * tan)
        A = ((k(4) * sec) * sec) * k(ipdl) + (k(2) * tt) * k(ipz)
        B = (k(-4) * tan) * k(ipz)
        C = k(f(2) * ipz)
        hb = B / k(2)
        b2 = hb * hb
        bb_y = k(3) / torch.sqrt(A - b2 / C)
        bb_z = k(3) / torch.sqrt(C - b2 / A)
        cx = ((z - k(tl_z)) / k(pw)).to(torch.int32)
        cy = ((k(tl_y) - y) / k(pw)).to(torch.int32)
        hw = (bb_z / k(pw) + k(0.5)).to(torch.int32)
        hh = (bb_y / k(pw) + k(0.5)).to(torch.int32)
        self.x0, self.x1 = (cx - hw).clamp(0, n_z - 1), (cx + hw).clamp(0, n_z - 1)
        self.y0, self.y1 = (cy - hh).clamp(0, n_y - 1), (cy + hh).clamp(0, n_y - 1)
        self.tan, self.sec, self.y, self.z, self.A, self.B, self.C = tan, sec, y, z, A, B, C
        self.tl_y_half, self.tl_z_half = k(tl_y - pw / f(2)), k(tl_z + pw / f(2))
        self.pw = k(pw)
        self.W = int((self.x1 - self.x0).max())
        self.H = int((self.y1 - self.y0).max())
        self.analytic = c.get("mode") == "gpu"
        self.index = torch.arange(len(zu), device=DEV)

    def of(self, subset, subsets):
        """The events of one ordered subset."""
        return self.index[subset::subsets]

    def blocks(self, events, sigmas=None):
        """(events, their pixels, kernel values, column and row terms) in blocks."""
        per = max(1, int(6e7 / max(1, self.W * self.H)))
        for i in range(0, len(events), per):
            yield self.block(events[i:i + per], sigmas)

    def block(self, e, sigmas):
        c = self.c
        v = lambda t: t[e][:, None, None]  # noqa: E731
        rows = v(self.y0) + torch.arange(self.H, device=DEV, dtype=torch.int32)[None, :, None]
        cols = v(self.x0) + torch.arange(self.W, device=DEV, dtype=torch.int32)[None, None, :]
        dy = (self.tl_y_half - rows.float() * self.pw) - v(self.y)
        dz = (self.tl_z_half + cols.float() * self.pw) - v(self.z)
        q = ((v(self.A) * dy) * dy + (v(self.B) * dy) * dz) + (self.C * dz) * dz
        ok = (q <= 9.0) & (rows < v(self.y1)) & (cols < v(self.x1))
        n, r, k = torch.nonzero(ok, as_tuple=True)
        del q, ok
        dy, dz = dy[n, r, 0].double(), dz[n, 0, k].double()
        pix = rows[n, r, 0].long() * c["n_z"] + cols[n, 0, k].long()
        tan, sec, y = (t[e][n].double() for t in (self.tan, self.sec, self.y))
        sz, sdl = sigmas or (float(np.float32(c["s_z"])), float(np.float32(c["s_dl"])))
        ipz, ipdl = 1 / sz ** 2, 1 / sdl ** 2
        kc = math.sqrt(ipz * ipz * ipdl) / (2 * math.pi ** 2)
        R = c["radius"]
        yp = dy + y
        ap, aq, ar = -(yp - R) * sec ** 2, -(yp + R) * sec ** 2, -2 * yp * sec * tan
        b, br = dz - dy * tan, -2 * dy * sec
        apq, arr = ipz * (ap * ap + aq * aq), ipdl * ar * ar
        norm, bib = apq + arr, 2 * ipz * b * b + ipdl * br * br
        if self.analytic:
            opq = -yp * sec * (1 + 2 * tan * tan)
            o_ic_b = ipz * (-(yp - R) * tan * sec ** 2 - (yp + R) * tan * sec ** 2) * b \
                + ipdl * opq * br
            b_ic_a = ipz * b * (ap + aq) + ipdl * br * ar
            norm = norm + 2 * o_ic_b
            value = kc / torch.sqrt(norm) * torch.exp(-0.5 * (bib - b_ic_a * b_ic_a / norm))
            return n, pix, value, None, None
        value = kc / torch.sqrt(norm) * torch.exp(-0.5 * bib)
        if not sigmas:
            return n, pix, value, None, None
        fz = (-2 + apq / norm + 2 * ipz * b * b) / sz
        fdl = (-1 + arr / norm + ipdl * br * br) / sdl
        return n, pix, value, fz, fdl

    def sensitivity(self):
        c = self.c
        p, n_y, n_z = c["pixel"], c["n_y"], c["n_z"]
        y = n_y * p / 2 - (torch.arange(n_y, device=DEV, dtype=torch.float64)[:, None] + 0.5) * p
        z = -n_z * p / 2 + (torch.arange(n_z, device=DEV, dtype=torch.float64)[None, :] + 0.5) * p

        def point(z, y):
            lp, lm = c["length"] / 2 + z, c["length"] / 2 - z
            rp, rm = c["radius"] + y, c["radius"] - y
            rp, rm = torch.where(rp <= 0, 1.0, rp), torch.where(rm <= 0, 1.0, rm)
            return (torch.atan(torch.minimum(lm / rm, lp / rp))
                    - torch.atan(torch.maximum(-lp / rm, -lm / rp))) / math.pi

        h = p / 2
        return (point(z, y) / 3 + (point(z + h, y + h) + point(z - h, y - h) + point(z - h, y + h)
                                   + point(z + h, y - h)) / 6).reshape(-1)

    def mlem(self, iterations, subsets):
        n_px = self.c["n_y"] * self.c["n_z"]
        rho = torch.ones(n_px, device=DEV, dtype=torch.float64)
        s = self.sensitivity() if self.analytic else torch.ones_like(rho)
        for _ in range(iterations):
            for sub in range(subsets):
                acc = torch.zeros_like(rho)
                for e in (b for b in [self.of(sub, subsets)] if len(b)):
                    for n, pix, k, _, _ in self.blocks(e):
                        d = torch.zeros(int(n[-1]) + 1 if len(n) else 0, device=DEV,
                                        dtype=torch.float64)
                        d.index_add_(0, n, k * rho[pix] * s[pix])
                        inv = torch.where(d > 0, 1 / d, torch.zeros_like(d))
                        acc.index_add_(0, pix, k * inv[n])
                rho = rho * acc * subsets
        return rho.reshape(self.c["n_y"], self.c["n_z"])


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        if sum(_evaluations(m) for m in _members(c)) > EXACT_MOST:
            return None
        return [_Strip64(m, _case_events(m, seed + 101 * i)).mlem(c["iterations"], 1)
                for i, m in enumerate(_members(c))]
    if _evaluations(c) > EXACT_MOST:
        return None
    if c["kind"] == "hybrid":
        return _hybrid64(c, seed)
    model = _Strip64(c, _case_events(c, seed))
    if c["kind"] != "project":
        return model.mlem(c["iterations"], c.get("subsets", 1))
    rho, w = (t.double() for t in _project_inputs(c, seed))
    sigmas = tuple(float(np.float32(v)) for v in ([0.9 * c["s_z"], 0.95 * c["s_dl"]] if c["sigma"]
                                                  else [c["s_z"], c["s_dl"]]))
    flat, y = rho.reshape(-1), torch.zeros_like(w)
    g = torch.zeros_like(flat)
    gs = torch.zeros(2, dtype=torch.float64, device=DEV)
    at = 0
    for n, pix, k, fz, fdl in model.blocks(model.index, sigmas):
        m = min(len(w) - at, max(1, int(6e7 / max(1, model.W * model.H))))
        kr = k * flat[pix]
        y[at:at + m].index_add_(0, n, kr)
        wn = w[at:at + m][n]
        g.index_add_(0, pix, k * wn)
        gs += torch.stack([(wn * kr * fz).sum(), (wn * kr * fdl).sum()])
        at += m
    g = g.reshape(c["n_y"], c["n_z"])
    return [y, g, gs] if c["sigma"] else [y, g]


def _evaluations(c):
    if c["kind"] == "hybrid":
        return 3 * c["iterations"] * c["responses"] * _voxels_per_event(c)
    return c["events"] * c.get("iterations", 1) * _pixels_per_event(c)


def _hybrid64(c, seed):
    """Frame events in binary32 as the scanner model defines them, then MLEM
    in binary64."""
    f = np.float32
    barrel, geo = _barrel_geometry(c["n_pix"])
    p, planes, z_left = _grid(c["n_pix"])
    first, second, zu, zd, dl = (torch.from_numpy(a).to(DEV) for a in _responses(c, barrel, seed))
    k = lambda v: torch.tensor(float(f(v)), device=DEV, dtype=torch.float32)  # noqa: E731
    seg, pos, w = (torch.from_numpy(geo[n]).to(DEV) for n in ("segments", "positions", "weights"))
    pix = torch.from_numpy(geo["pixels"]).to(DEV).long()
    lb, le = (torch.from_numpy(geo[n]).to(DEV) for n in ("lor_begin", "lor_end"))
    flat = pix[:, 0] + c["n_pix"] * pix[:, 1]
    sens = torch.zeros(c["n_pix"] ** 2, device=DEV, dtype=torch.float64)
    sens = sens.index_add_(0, flat, w.double()).float()
    w = w / sens[flat]
    dx, dy = seg[:, 2] - seg[:, 0], seg[:, 3] - seg[:, 1]
    length = torch.sqrt(dx * dx + dy * dy)
    mid = (seg[:, :2] + seg[:, 2:]) / k(2)
    direction = torch.stack([dx / length, dy / length], 1)
    li = first.long() * (first.long() + 1) // 2 + second.long()
    R = length[li] / k(2)
    ipz, ipdl = f(1) / (f(H_SIGMA_Z) * f(H_SIGMA_Z)), f(1) / (f(H_SIGMA_DL) * f(H_SIGMA_DL))
    tan = (zu - zd) / (k(2) * R)
    sec = torch.sqrt(k(1) + tan * tan)
    up = k(-0.5) * (dl / sec)
    right = k(0.5) * ((zu + zd) + (k(2) * up) * tan)
    A = ((k(4) * sec) * sec) * k(ipdl) + (k(2) * (tan * tan)) * k(ipz)
    B = (k(-4) * tan) * k(ipz)
    C = k(f(2) * ipz)
    b2 = (B / k(2)) * (B / k(2))
    half_up, half_right = k(3) / torch.sqrt(A - b2 / C), k(3) / torch.sqrt(C - b2 / A)
    plane = lambda z: ((z - k(z_left)) / k(p)).to(torch.int32)  # noqa: E731
    pb = plane(right - half_right).clamp_min(0).long()
    pe = (plane(right + half_right) + 1).clamp_max(planes).long()
    t_up = ((up + half_up) + R) / (k(2) * R)
    t_dn = ((up - half_up) + R) / (k(2) * R)
    lor_of = torch.repeat_interleave(torch.arange(len(lb), device=DEV), le - lb)
    keys = lor_of * 4.0 + pos.double()
    find = lambda t, right: torch.searchsorted(  # noqa: E731
        keys, li * 4.0 + t.double().clamp(-1, 2), right=right)
    ib = torch.minimum(torch.maximum(find(t_dn, False), lb[li]), le[li])
    ie = torch.minimum(torch.maximum(find(t_up, True), lb[li]), le[li]) + 1
    ie = ie.clamp_max(len(pos))
    keep = torch.nonzero((pe > 0) & (pb < planes) & (ie > ib))[:, 0]
    n_vox = ((ie - ib) * (pe - pb).clamp_min(0))[keep]
    groups = torch.split(keep, max(1, int(2e7 / max(1.0, float(n_vox.float().mean())))))
    # pixel centres as the grid defines them (binary32)
    p32 = f(p)
    llc = -p32 * f(c["n_pix"]) / f(2) + p32 / f(2)
    centre = k(llc) + torch.arange(c["n_pix"], device=DEV).float() * k(p32)
    zc = (torch.arange(planes, device=DEV).float() + k(0.5)) * k(p32) + k(z_left)
    n_px = c["n_pix"] ** 2
    rho = torch.ones(planes * n_px, device=DEV, dtype=torch.float64)
    ipz, ipdl = float(ipz), float(ipdl)
    norm_c = math.sqrt(ipz * ipz * ipdl) / (2 * math.pi ** 2)
    half_L = LENGTH / 2
    for _ in range(c["iterations"]):
        acc = torch.zeros_like(rho)
        for e in groups:
            npl = (pe - pb)[e]
            cnt = (ie - ib)[e] * npl
            n = torch.repeat_interleave(torch.arange(len(e), device=DEV), cnt)
            o = torch.arange(len(n), device=DEV) - (torch.cumsum(cnt, 0) - cnt)[n]
            ev = e[n]
            info, iz = ib[ev] + o // npl[n], pb[ev] + o % npl[n]
            l, px = li[ev], pix[info]
            upp = ((centre[px[:, 0]] - mid[l, 0]) * direction[l, 0]
                   + (centre[px[:, 1]] - mid[l, 1]) * direction[l, 1]).double()
            z, Rd = zc[iz].double(), R[ev].double()
            t, s = tan[ev].double(), sec[ev].double()
            d_up = upp - up[ev].double()
            ap, aq, ar = -(upp - Rd) * s ** 2, -(upp + Rd) * s ** 2, -2 * upp * s * t
            b, br = z - right[ev].double() - d_up * t, -2 * d_up * s
            val = norm_c / torch.sqrt(ipz * (ap * ap + aq * aq) + ipdl * ar * ar) \
                * torch.exp(-0.5 * (2 * ipz * b * b + ipdl * br * br))
            lm, lp = half_L - z, half_L + z
            view = (torch.atan(torch.minimum(lm / (Rd - upp), lp / (Rd + upp)))
                    - torch.atan(torch.maximum(-lp / (Rd - upp), -lm / (Rd + upp)))) / math.pi
            fl = flat[info]
            vox = fl + iz * n_px
            weight = torch.where(view > 0, val / view, torch.zeros_like(val)) \
                * w[info].double() * rho[vox]
            d = torch.zeros(len(e), device=DEV, dtype=torch.float64)
            d.index_add_(0, n, weight * sens[fl].double())
            inv = torch.where(d > 0, 1 / d, torch.zeros_like(d))
            acc.index_add_(0, vox, weight * inv[n])
        rho = acc
    return rho.reshape(planes, c["n_pix"], c["n_pix"])
