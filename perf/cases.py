"""The calls this engine is used for, as cases that can be timed and checked.

A case is one call (or one short sequence of calls) that a program makes through
the public Python bindings of the C-ABI: a projection or back projection of one
image, of a set of images, of a cone-beam volume, and Ambrosio-Tortorelli
reconstructions alone and in batches.  Sizes are the benchmark workloads' own
(medimage_gb300/configs.py, bench.py) and sizes between and beside them.

Inputs are seeded synthetic scans.  Sinograms are closed-form line integrals of
the ellipses (ellipsoids) with Poisson counting noise, so they do not depend on
any projector.  `exact` evaluates the same call in 64 bits with plain torch.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import torch

import medimage_gb300 as mg

DEV = "cuda"
SOD, SDD = 541.0, 949.0  # fan-beam source and detector distances (mm)
# GoldenC's weights and ten edge iterations.  Four image iterations an outer iteration, not its ten: past five, the
# line searches after a median step divide nearly cancelling sums, and any rounding moves f by up to 1e-4.
AT = dict(alpha=1000.0, beta=0.002, epsilon=1e-4, iter_image=4, iter_edge=10)
STOP = 0.05              # the tracers end a ray once less than this is left of it (mm; voxels for the cone beam)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a quick look at a coarse grid; latency and launches
        dict(name="forward_64", kind="project", op="forward", n=64, views=90, dets=128),
        # a region of interest: odd image, ragged tiles, view and detector blocks
        dict(name="back_217_odd", kind="project", op="back", n=217, views=301, dets=390),
        # the flagship slice (512^2, 720 views x 888 detectors), one projection
        dict(name="forward_512", kind="project", op="forward", n=512, views=720, dets=888),
        # the same slice, one back projection of its measured sinogram
        dict(name="back_512", kind="project", op="back", n=512, views=720, dets=888),
        # the largest slices that are served: 1024^2, 1440 views x 1536 detectors
        dict(name="back_1024", kind="project", op="back", n=1024, views=1440, dets=1536),
        # slices of one scanner projected together (two groups of four)
        dict(name="set_forward_8x512", kind="set", op="forward", slices=8, mix=False, n=512, views=720, dets=888),
        # uneven scans in one set: a group of three, a pair, one alone and a
        # non-uniform view table (a ray table)
        dict(name="set_back_mixed_384", kind="set", op="back", slices=7, mix=True, n=384, views=540, dets=768),
        # one small slice from host memory to host memory in one call (the
        # linear mode), creation of the solver included
        dict(name="reconstruct_256_host", kind="solve", slices=1, mix=False, host=True, linear=True, outer=2,
             n=256, views=360, dets=512),
        # the benchmark's batch: 16 slices of one scanner, resident, exact mode
        dict(name="solve_16x512", kind="solve", slices=16, mix=False, host=False, linear=False, outer=2,
             n=512, views=720, dets=888),
        # a batch of uneven scans (the shapes of the 64-slice workload)
        dict(name="solve_mixed_7x256", kind="solve", slices=7, mix=True, host=False, linear=False, outer=2,
             n=256, views=360, dets=512),
        # cone beam: one projection of a volume
        dict(name="cone_forward_256", kind="cone", op="forward", n=256, nz=256, views=180, rows=192, cols=256),
        # cone beam, odd sizes: one back projection of a measured sinogram
        dict(name="cone_back_201_odd", kind="cone", op="back", n=201, nz=161, views=121, rows=150, cols=203),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; its work stays below the largest listed one's."""
    kind = rng.choice(["project", "project", "project", "set", "set", "solve", "solve", "cone"])
    if kind == "cone":
        n = _log(rng, 40, 256)
        return dict(kind=kind, op=rng.choice(["forward", "back"]), n=n, nz=max(8, int(n * rng.uniform(0.4, 1.0))),
                    views=rng.randint(24, 180), rows=max(16, int(n * rng.uniform(0.5, 0.8))),
                    cols=max(16, int(n * rng.uniform(0.8, 1.05))))
    top = {"project": 1024, "set": 640, "solve": 512}[kind]
    n = _log(rng, 48, top)
    views = max(24, int(n * rng.uniform(1.0, 1.45)))
    dets = 2 * max(16, int(n * rng.uniform(0.75, 1.0)))
    c = dict(kind=kind, n=n, views=views, dets=dets)
    if kind == "project":
        return dict(c, op=rng.choice(["forward", "back"]))
    c.update(slices=rng.randint(2, 9), mix=rng.random() < 0.5)
    if kind == "set":
        return dict(c, op=rng.choice(["forward", "back"]))
    host = rng.random() < 0.3
    return dict(c, slices=1 if host else c["slices"], mix=c["mix"] and not host, host=host,
                linear=rng.random() < 0.4, outer=rng.randint(1, 2))


# ---------------------------------------------------------------- geometries
def _pixel(n):
    return 384.0 / n  # the benchmark's field of view is 384 mm at every grid size


def _geometries(case):
    """The fan geometries (or view tables) of the case's slices, in order; slices of one scanner share an entry."""
    n, v, d = case["n"], case["views"], case["dets"]
    main = ("fan", n, v, d)
    k = case.get("slices", 1)
    if not case.get("mix"):
        return [main] * k
    half = max(24, 2 * (n // 3))
    second = ("fan", half, max(24, v // 2), 2 * max(16, d // 3))
    third = ("fan", max(24, n - 37), max(24, v - 11), max(32, d - 102))
    table = ("table", half, max(24, v // 3), 2 * max(16, d // 4))
    order = [main, second, main, third, main, second, table]
    return (order + [main, third])[:k]


def _angles(geom):
    """Source angles in degrees, FP64."""
    kind, n, v, d = geom
    if kind == "fan":
        step = 360.0 / v
        return [i * step for i in range(v)]
    return [360.0 * (i + 0.3 * math.sin(0.7 * i)) / v for i in range(v)]  # uneven steps


def _pitch(geom):
    n, d = geom[1], geom[3]
    r = n * _pixel(n) * math.sqrt(2.0) / 2.0
    return 2.0 * math.degrees(math.asin(r / SOD)) / d


def _plan(geom):
    kind, n, v, d = geom
    if kind == "fan":
        return mg.Plan.fan(mg.engine.FanGeometry.covering(n, _pixel(n), v, d, SOD, SDD))
    return mg.Plan.rays(mg.RayGeometry.fan_from_view_table(n, _pixel(n), d, _angles(geom), SOD, SDD, _pitch(geom)))


def _rays(geom, lo=0, hi=None):
    """Source, unit direction and length (mm) of the rays lo..hi of the flattened sinogram, FP64."""
    kind, n, v, d = geom
    hi = v * d if hi is None else hi
    i = torch.arange(lo, hi, device=DEV)
    a = torch.tensor(_angles(geom), dtype=torch.float64, device=DEV)[i // d] / 180.0 * math.pi
    t = ((i % d) - d // 2 + 0.5).double() * (_pitch(geom) * math.pi / 180.0) + math.pi + a
    half = n * _pixel(n) / 2.0
    return SOD * a.cos() + half, SOD * a.sin() + half, t.cos(), t.sin(), SDD


def _cone(case):
    n = case["n"]
    # the benchmark's field of view: 102.4 mm across, on a 256 mm wide detector that sees all of it
    return dict(nx=n, ny=n, nz=case["nz"], voxel_mm=102.4 / n, nproj=case["views"], ndx=case["rows"],
                ndy=case["cols"], pitch_mm=256.0 / case["cols"], sod_mm=600.0, sdd_mm=1000.0)


def _cone_rays(g, lo, hi):
    """Source, unit direction and length (voxels) of the rays lo..hi, FP64."""
    g = SimpleNamespace(**g)
    i = torch.arange(lo, hi, device=DEV)
    view, rem = i // (g.ndx * g.ndy), i % (g.ndx * g.ndy)
    th = view.double() / g.nproj * 2.0 * math.pi
    c, s = th.cos(), th.sin()
    vx, pt = float(torch.tensor(g.voxel_mm, dtype=torch.float32)), float(torch.tensor(g.pitch_mm, dtype=torch.float32))
    dx = (rem % g.ndy - g.ndy // 2 + 0.5).double() * pt
    dz = (g.ndx // 2 - rem // g.ndy - 0.5).double() * pt
    dy = g.sdd_mm - g.sod_mm
    sx, sy = s * g.sod_mm / vx + g.nx / 2.0, -c * g.sod_mm / vx + g.nx / 2.0
    ex, ey, ez = (c * dx - s * dy) / vx + g.nx / 2.0, (s * dx + c * dy) / vx + g.nx / 2.0, dz / vx + g.nz / 2.0
    sz = torch.full_like(sx, g.nz / 2.0)
    ux, uy, uz = ex - sx, ey - sy, ez - sz
    L = (ux * ux + uy * uy + uz * uz).sqrt()
    return (sx, sy, sz), (ux / L, uy / L, uz / L), L


# -------------------------------------------------------------------- inputs
def _gen(seed, k=0):
    return torch.Generator(device="cpu").manual_seed(seed * 1009 + k)


def _ellipses(gen, dim):
    """A head-like section: a shell, its content and two dozen smaller structures; attenuation in 1/mm.
    Rows of (value, semi-axes, centre, angle in the first two axes), in units of half the field of view."""
    def u(lo, hi, m=1):
        return torch.rand(m, generator=gen, dtype=torch.float64) * (hi - lo) + lo
    rows = [(0.02, [0.69, 0.92, 0.8], [0.0, 0.0, 0.0], 0.0), (-0.016, [0.66, 0.87, 0.75], [0.0, -0.02, 0.0], 0.0)]
    for _ in range(24):
        r, t = float(u(0, 0.5)), float(u(0, 2 * math.pi))
        rows.append((float(u(-0.003, 0.004)), u(0.02, 0.2, 3).tolist(),
                     [r * math.cos(t), r * math.sin(t), float(u(-0.4, 0.4))], float(u(0, math.pi))))
    return [(a, ax[:dim], c[:dim], t) for a, ax, c, t in rows]


def _image(n, seed, k):
    c = (torch.arange(n, dtype=torch.float64, device=DEV) + 0.5 - n / 2.0) / (n / 2.0)
    X, Y = c[:, None], c[None, :]
    out = torch.zeros(n, n, dtype=torch.float64, device=DEV)
    for a, ax, ce, t in _ellipses(_gen(seed, k), 2):
        x = (X - ce[0]) * math.cos(t) + (Y - ce[1]) * math.sin(t)
        y = (Y - ce[1]) * math.cos(t) - (X - ce[0]) * math.sin(t)
        out += a * ((x / ax[0]) ** 2 + (y / ax[1]) ** 2 <= 1.0)
    return out.clamp_(min=0.0).float()


def _volume(case, seed):
    g = SimpleNamespace(**_cone(case))
    c = (torch.arange(g.nx, dtype=torch.float64, device=DEV) + 0.5 - g.nx / 2.0) / (g.nx / 2.0)
    z = (torch.arange(g.nz, dtype=torch.float64, device=DEV) + 0.5 - g.nz / 2.0) / (g.nz / 2.0)
    Z, X, Y = z[:, None, None], c[None, :, None], c[None, None, :]
    out = torch.zeros(g.nz, g.nx, g.nx, dtype=torch.float32, device=DEV)
    for a, ax, ce, t in _ellipses(_gen(seed), 3):
        x = (X - ce[0]) * math.cos(t) + (Y - ce[1]) * math.sin(t)
        y = (Y - ce[1]) * math.cos(t) - (X - ce[0]) * math.sin(t)
        out += a * ((x / ax[0]) ** 2 + (y / ax[1]) ** 2 + ((Z - ce[2]) / ax[2]) ** 2 <= 1.0)
    return out.clamp_(min=0.0)


def _chords(rows, src, dirs, scale, shape, gen, i0=5e3):
    """Noisy line integrals: the closed-form chords through the ellipses (ellipsoids), Poisson counts of i0 photons."""
    total = torch.zeros(shape, dtype=torch.float64, device=DEV).reshape(-1)
    for a, ax, ce, t in rows:
        cs, sn = math.cos(t), math.sin(t)
        p = [s - o - c * o for s, o, c in zip(src, scale, ce)]  # relative to the centre, in the grid's unit
        p = [p[0] * cs + p[1] * sn, p[1] * cs - p[0] * sn] + p[2:]
        d = [dirs[0] * cs + dirs[1] * sn, dirs[1] * cs - dirs[0] * sn] + list(dirs[2:])
        w = [1.0 / (e * o) for e, o in zip(ax, scale)]
        A = sum((di * wi) ** 2 for di, wi in zip(d, w))
        B = sum(pi * di * wi * wi for pi, di, wi in zip(p, d, w))
        C = sum((pi * wi) ** 2 for pi, wi in zip(p, w)) - 1.0
        total += a * 2.0 * (B * B - A * C).clamp_(min=0.0).sqrt() / A
    lam = (i0 * torch.exp(-total.clamp_(min=0.0))).float()
    g = torch.Generator(device=DEV).manual_seed(int(torch.randint(1 << 30, (1,), generator=gen)))
    counts = torch.poisson(lam, generator=g).clamp_(min=1.0)
    return (-(counts / i0).log()).reshape(shape).contiguous()


def _sinogram(geom, seed, k):
    kind, n, v, d = geom
    gen = _gen(seed, 7000 + k)
    half = n * _pixel(n) / 2.0
    sx, sy, dx, dy, _ = _rays(geom)
    return _chords(_ellipses(gen, 2), [sx, sy], [dx, dy], [half, half], (v, d), gen)


def _cone_sinogram(case, seed):
    gen = _gen(seed, 9000)
    shape = (case["views"], case["rows"], case["cols"])
    src, dirs, _ = _cone_rays(_cone(case), 0, math.prod(shape))
    half = [case["n"] / 2.0, case["n"] / 2.0, case["nz"] / 2.0]
    # voxel units: the attenuation of a voxel edge
    rows = [(a * 102.4 / case["n"], ax, c, t) for a, ax, c, t in _ellipses(gen, 3)]
    return _chords(rows, list(src), list(dirs), half, shape, gen)


def _inputs(case, seed):
    if case["kind"] == "cone":
        return [(_volume if case["op"] == "forward" else _cone_sinogram)(case, seed)]
    geoms = _geometries(case)
    if case.get("op") == "forward":
        return [_image(g[1], seed, k) for k, g in enumerate(geoms)]
    return [_sinogram(g, seed, k) for k, g in enumerate(geoms)]


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    """The inputs on the GPU (host memory for the host call), the plans of the geometries, and the solver or
    projection set that such a program makes once."""
    kind = case["kind"]
    s = dict(case=case, inputs=_inputs(case, seed))
    if kind == "cone":
        s["plans"] = [mg.Plan.cone(mg.ConeGeometry(**_cone(case)))]
    else:
        geoms = _geometries(case)
        made = {g: _plan(g) for g in dict.fromkeys(geoms)}
        s["plans"] = [made[g] for g in geoms]
    if kind == "solve":
        prm = s["params"] = mg.Params(iter_alt=case["outer"], mode=1 if case["linear"] else 0, **AT)
        if case["host"]:
            s["inputs"] = [x.cpu().numpy() for x in s["inputs"]]
            return s
        s["solver"] = mg.Solver(s["plans"], prm)
        s["outputs"] = [[torch.empty(p.img_shape, device=DEV) for p in s["plans"]] for _ in range(2)]
        return s
    shapes = [p.sino_shape if case["op"] == "forward" else p.img_shape for p in s["plans"]]
    s["outputs"] = [torch.empty(shape, device=DEV) for shape in shapes]
    if kind == "set":
        s["set"] = mg.ProjSet(s["plans"])
    return s


def run(s):
    case = s["case"]
    st = torch.cuda.current_stream().cuda_stream
    if case["kind"] == "solve":
        if case["host"]:
            f, v = mg.reconstruct(s["plans"][0], s["params"], s["inputs"][0])
            return {"f": f, "v": v}
        solver, (fs, vs) = s["solver"], s["outputs"]
        for i, x in enumerate(s["inputs"]):
            solver.set_sino_dev(i, x.data_ptr(), st)
        solver.run(st, sync=False)
        for i in range(len(fs)):
            rc = mg.lib().at_solver_get(solver.handle, i, fs[i].data_ptr(), vs[i].data_ptr(), st)
            if rc != 0:
                raise mg.AtError("at_solver_get", rc, mg.lib().at_last_error().decode())
        return {"f": fs, "v": vs}
    forward = case["op"] == "forward"
    if case["kind"] == "set":
        call = s["set"].forward_dev if forward else s["set"].back_dev
        call([x.data_ptr() for x in s["inputs"]], [y.data_ptr() for y in s["outputs"]], st)
        return s["outputs"]
    plan, x, y = s["plans"][0], s["inputs"][0], s["outputs"][0]
    (plan.forward_dev if forward else plan.back_dev)(x.data_ptr(), y.data_ptr(), st)
    return y


def work(case):
    """Inputs read once, outputs written once (the traversal can be recomputed), and a multiply-add for each pixel
    (voxel) that a ray crosses, about 0.88 n of them a ray (1.2 n where the cone beam meets the volume)."""
    if case["kind"] == "cone":
        vox, rays = case["n"] ** 2 * case["nz"], case["views"] * case["rows"] * case["cols"]
        return {"bytes": 4 * (vox + rays), "flops": 2 * 1.2 * rays * case["n"]}
    total, passes, per_pixel = 0.0, 1, 1
    if case["kind"] == "solve":  # 11 forward and 4 back projections an outer iteration; 6 + 4 in linear mode
        passes, per_pixel = case["outer"] * (10 if case["linear"] else 15), 2
    nbytes = 0
    for _, n, v, d in _geometries(case):
        total += 2 * 0.88 * n * v * d * passes
        nbytes += 4 * (per_pixel * n * n + v * d)
    return {"bytes": nbytes, "flops": total}


# ------------------------------------------------- the same calls in 64 bits
def _segments(n, px, src, dirs, L):
    """Pixels and lengths of rays through the n x n grid, two per row of the axis a ray runs along: (index, length)
    pairs of shape [rays, n].  A ray's last piece is left out when less than STOP of the ray is left where it begins."""
    (sx, sy), (dx, dy) = src, dirs
    swap = dy.abs() > dx.abs()
    su, sv = torch.where(swap, sy, sx), torch.where(swap, sx, sy)
    du, dv = torch.where(swap, dy, dx), torch.where(swap, dx, dy)
    ext = n * px
    far = torch.full_like(du, 1e30)

    def span(s, d):
        inv = torch.where(d == 0, far, 1.0 / d)
        a, b = -s * inv, (ext - s) * inv
        return torch.minimum(a, b), torch.maximum(a, b)
    (u0, u1), (v0, v1) = span(su, du), span(sv, dv)
    lmin = torch.maximum(u0, v0).clamp_(min=0.0)
    lmax = torch.maximum(torch.minimum(u1, v1).clamp_(max=L), lmin)
    i = torch.arange(n, dtype=torch.float64, device=DEV)
    a = (i * px - su[:, None]) / du[:, None]
    b = ((i + 1) * px - su[:, None]) / du[:, None]
    lo, hi = torch.maximum(torch.minimum(a, b), lmin[:, None]), torch.minimum(torch.maximum(a, b), lmax[:, None])
    del a, b
    hi = torch.maximum(hi, lo)
    y = (sv[:, None] + lo * dv[:, None]) / px
    plane = torch.where(dv[:, None] > 0, y.floor() + 1, y.ceil() - 1)
    cut = torch.where(dv[:, None] == 0, far[:, None], (plane * px - sv[:, None]) / dv[:, None])
    cut = torch.minimum(torch.maximum(cut, lo), hi)
    del y, plane
    out = []
    for p, q in ((lo, cut), (cut, hi)):
        c = ((sv[:, None] + 0.5 * (p + q) * dv[:, None]) / px).floor().long().clamp_(0, n - 1)
        w = (q - p) * (p < (lmax[:, None] - STOP))
        r = torch.arange(n, device=DEV)[None, :]
        out.append((torch.where(swap[:, None], c * n + r, r * n + c), w))
    return out


class _Matrix:
    """The projector of one geometry in 64 bits; small ones are kept, large ones are traced anew for each product."""

    def __init__(self, geom):
        self.geom, self.n = geom, geom[1]
        self.rays = geom[2] * geom[3]
        self.step = max(1, (1 << 24) // self.n)
        self.kept = [self._piece(lo) for lo in range(0, self.rays, self.step)] if self.rays * self.n <= 1 << 27 else None

    def _piece(self, lo):
        sx, sy, dx, dy, L = _rays(self.geom, lo, min(self.rays, lo + self.step))
        return _segments(self.n, _pixel(self.n), (sx, sy), (dx, dy), L)

    def _pieces(self):
        for k, lo in enumerate(range(0, self.rays, self.step)):
            yield lo, self.kept[k] if self.kept else self._piece(lo)

    def forward(self, img):
        out, flat = torch.empty(self.rays, dtype=torch.float64, device=DEV), img.reshape(-1)
        for lo, parts in self._pieces():
            s = sum((flat[i] * w).sum(1) for i, w in parts)
            out[lo:lo + s.numel()] = s
        return out.reshape(self.geom[2], self.geom[3])

    def back(self, sino):
        out, flat = torch.zeros(self.n * self.n, dtype=torch.float64, device=DEV), sino.reshape(-1)
        for lo, parts in self._pieces():
            for i, w in parts:
                out.index_add_(0, i.reshape(-1), (w * flat[lo:lo + w.shape[0], None]).reshape(-1))
        return out.reshape(self.n, self.n)


def _pad(a, value):
    return torch.nn.functional.pad(a, (1, 1, 1, 1), value=value)


def _median(a):
    p = _pad(a, 0.0)
    n = a.shape[0]
    return torch.stack([p[i:i + n, j:j + n] for i in range(3) for j in range(3)]).median(0).values


def _smooth(u, v, alpha, eps):
    """The stencil alpha div((v^2 + 0.01 eps^2) grad u) and its energy over the interior."""
    P, T, e2 = _pad(v, 1.0), _pad(u, 0.0), 0.01 * eps * eps
    c, up, lf = P[1:-1, 1:-1] ** 2, P[:-2, 1:-1] ** 2, P[1:-1, :-2] ** 2
    t, tu, td, tl, tr = u, T[:-2, 1:-1], T[2:, 1:-1], T[1:-1, :-2], T[1:-1, 2:]
    st = c * (td - t) + c * (tr - t) - up * (t - tu) - lf * (t - tl) + e2 * (td + tr - 4 * t + tu + tl)
    en = alpha * (c + e2) * ((t - tu) ** 2 + (t - tl) ** 2)
    return alpha * st, float(en[1:-1, 1:-1].sum())


def _image_step(A, g, f, v, prm):
    u = f.clone()
    r = g - A.forward(u)
    st, en = _smooth(u, v, prm.alpha, prm.epsilon)
    d = A.back(r) + st
    old = float((r * r).sum()) + en
    p = d.clone()
    e2, K = 0.01 * prm.epsilon ** 2, prm.iter_image
    for k in range(1, K + 1):
        q = A.forward(p)
        T = _pad(p, 0.0)
        nv = float(((v * v + e2) * ((p - T[:-2, 1:-1]) ** 2 + (p - T[1:-1, :-2]) ** 2)).sum())
        qq = float((q * q).sum())
        c1 = float((p * d).sum()) / (qq + prm.alpha * nv)
        before = u
        u = u + c1 * p
        if k % (K // 2) == 0:
            u = _median(u)
        if k == K or float((c1 * p).abs().max()) < 1e-5:
            return u
        e = A.forward(u) - g
        st, en = _smooth(u, v, prm.alpha, prm.epsilon)
        new = float((e * e).sum()) + en
        if 1.1 * old < new and k > 1:
            return before
        old = new
        r = r - c1 * q
        d = A.back(r) + st
        p = d - float((A.forward(d) * q).sum()) / qq * p
    return u


def _edge_step(f, v, prm):
    F = _pad(f, 0.0)
    nn = (0.5 * (F[2:, 1:-1] - F[:-2, 1:-1])) ** 2 + (0.5 * (F[1:-1, 2:] - F[1:-1, :-2])) ** 2
    b, e = prm.beta, prm.epsilon
    for k in range(1, prm.iter_edge + 1):
        T = _pad(v, 1.0)
        lap = 0.25 * (T[2:, 1:-1] + T[1:-1, 2:] - 4 * v + T[:-2, 1:-1] + T[1:-1, :-2])
        d = -(prm.alpha * v * nn - b * e * lap + b * (v - 1) / (4 * e))
        D = _pad(d, 0.0)
        grad = ((0.5 * (D[2:, 1:-1] - D[:-2, 1:-1])) ** 2 + (0.5 * (D[1:-1, 2:] - D[1:-1, :-2])) ** 2).sum()
        nd = (d * d).sum()
        c = float(nd / (prm.alpha * (nn * d * d).sum() + b * e * grad + b / (4 * e) * nd))
        v = (v + c * d).clamp(0.0, 1.0)
        if float((c * d).abs().max()) < 1e-5:
            break
    return v


def _solve(A, g, prm):
    f = torch.zeros(A.n, A.n, dtype=torch.float64, device=DEV)
    v = torch.ones_like(f)
    for _ in range(prm.iter_alt):
        f = _image_step(A, g, f, v, prm)
        v = _edge_step(f, v, prm)
    return f, v


def _cone_segments(g, lo, hi):
    """Voxels and lengths of the rays lo..hi, three per slab of the axis a ray runs along: pairs of [rays, n]."""
    (sx, sy, sz), (dx, dy, dz), L = _cone_rays(g, lo, hi)
    n, nz = g["nx"], g["nz"]
    swap = dy.abs() > dx.abs()
    su, sv = torch.where(swap, sy, sx), torch.where(swap, sx, sy)
    du, dv = torch.where(swap, dy, dx), torch.where(swap, dx, dy)
    far = torch.full_like(du, 1e30)

    def span(s, d, m):
        inv = torch.where(d == 0, far, 1.0 / d)
        a, b = -s * inv, (m - s) * inv
        return torch.minimum(a, b), torch.maximum(a, b)
    spans = [span(su, du, n), span(sv, dv, n), span(sz, dz, nz)]
    lmin = torch.maximum(torch.maximum(spans[0][0], spans[1][0]), spans[2][0]).clamp_(min=0.0)
    lmax = torch.minimum(torch.minimum(spans[0][1], spans[1][1]), torch.minimum(spans[2][1], L))
    lmax = torch.maximum(lmax, lmin)
    i = torch.arange(n, dtype=torch.float64, device=DEV)
    a, b = (i - su[:, None]) / du[:, None], (i + 1 - su[:, None]) / du[:, None]
    p0, p3 = torch.maximum(torch.minimum(a, b), lmin[:, None]), torch.minimum(torch.maximum(a, b), lmax[:, None])
    del a, b
    p3 = torch.maximum(p3, p0)

    def cut(s, d):
        y = s[:, None] + p0 * d[:, None]
        plane = torch.where(d[:, None] > 0, y.floor() + 1, y.ceil() - 1)
        c = torch.where(d[:, None] == 0, far[:, None], (plane - s[:, None]) / d[:, None])
        return torch.minimum(torch.maximum(c, p0), p3)
    cv, cz = cut(sv, dv), cut(sz, dz)
    p1, p2 = torch.minimum(cv, cz), torch.maximum(cv, cz)
    r = torch.arange(n, device=DEV)[None, :]
    out = []
    for p, q in ((p0, p1), (p1, p2), (p2, p3)):
        mid = 0.5 * (p + q)
        c = (sv[:, None] + mid * dv[:, None]).floor().long().clamp_(0, n - 1)
        z = (sz[:, None] + mid * dz[:, None]).floor().long().clamp_(0, nz - 1)
        w = (q - p) * (p < (lmax[:, None] - STOP))
        out.append((z * n * n + torch.where(swap[:, None], c * n + r, r * n + c), w))
    return out


def _cone_exact(case, x):
    g, forward, n = _cone(case), case["op"] == "forward", case["n"]
    shape = (case["views"], case["rows"], case["cols"]) if forward else (case["nz"], n, n)
    rays, flat = case["views"] * case["rows"] * case["cols"], x.double().reshape(-1)
    out = torch.zeros(math.prod(shape), dtype=torch.float64, device=DEV)
    step = max(1, (1 << 25) // n)
    for lo in range(0, rays, step):
        hi = min(rays, lo + step)
        for i, w in _cone_segments(g, lo, hi):
            if forward:
                out[lo:hi] += (flat[i] * w).sum(1)
            else:
                out.index_add_(0, i.reshape(-1), (w * flat[lo:hi, None]).reshape(-1))
    return out.reshape(shape)


def exact(case, seed):
    x = _inputs(case, seed)
    if case["kind"] == "cone":
        return _cone_exact(case, x[0])
    geoms = _geometries(case)
    if case["kind"] == "solve":
        # a batch of full-size slices takes minutes in 64 bits
        if sum(n * v * d for _, n, v, d in geoms) * case["outer"] > 1 << 30:
            return None
        prm = SimpleNamespace(iter_alt=case["outer"], **AT)
        made = {g: _Matrix(g) for g in dict.fromkeys(geoms)}
        fv = [_solve(made[g], s.double(), prm) for g, s in zip(geoms, x)]
        if case["host"]:
            return {"f": fv[0][0], "v": fv[0][1]}
        return {"f": [f for f, _ in fv], "v": [v for _, v in fv]}
    made = {g: _Matrix(g) for g in dict.fromkeys(geoms)}
    ys = [made[g].forward(s.double()) if case["op"] == "forward" else made[g].back(s.double())
          for g, s in zip(geoms, x)]
    return ys if case["kind"] == "set" else ys[0]
