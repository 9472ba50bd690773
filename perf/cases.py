"""Timed cases of the projection and reconstruction path.

Each case is one call a user's program makes (a projection, one OSEM
sub-iteration, a whole reconstruction, a gradient, a batch) on a scanner, a
volume and data of stated sizes.  Scanners are rings of point crystals; the
measured data are Poisson counts of an attenuated elliptical body with a hot
insert, made from the chord lengths of the lines of response, so they come
from the seed alone and need no projector.

``exact`` traces the same paths in plain torch, in 64 bits: FIR's rules for
entry, ties (1e-5 in the path parameter) and voxel extents, with every sum in
double.
"""
import math

import numpy as np
import torch

from fir_b200 import autograd, capi, workloads
from fir_b200.geometry import OSEMParams, ProjSpec, ScannerSpec, VolSpec

EPS = 1e-5

# Fields every case has; a case names what differs.
BASE = dict(kind="forward", rings=32, crystals=512, radius=400.0, pitch=4.0, tang=125, span=1,
            nx=200, ny=200, nz=64, vx=3.0, vz=3.0, subsets=16, iterations=1, frames=1, dtype="float32",
            counts=5e8, bias=False, mult=False, skip_zero=False, deterministic=False, cut=0.0, fwhm=4.0,
            problems=1)


def _case(name, **kw):
    c = dict(BASE)
    c.update(kw)
    c["name"] = name
    return c


def listed():
    return [
        # the least work a call can bring: a sub-iteration of a preclinical-sized
        # test scanner, where launches and latency are what counts
        _case("tiny_subiteration", kind="subiteration", rings=4, crystals=64, radius=120.0, tang=21,
              nx=32, ny=32, nz=8, vx=4.0, vz=4.0, subsets=4, counts=1e5),
        # a whole small reconstruction in one call: 8 rings x 128 crystals, 4
        # subsets x 3 iterations with the filter, randoms as a bias
        _case("small_osem", kind="osem", rings=8, crystals=128, radius=200.0, tang=43,
              nx=64, ny=64, nz=16, vx=4.0, vz=4.0, subsets=4, iterations=3, counts=1e6, bias=True),
        # the same scanner's projector and its gradient in 64 bits, two
        # frames: gradient checks
        _case("small_gradient_f64", kind="gradient", rings=8, crystals=128, radius=200.0, tang=43,
              nx=61, ny=67, nz=15, vx=4.0, vz=4.0, frames=2, dtype="float64", counts=1e6),
        # attenuation factors of a mid-sized scanner from its mu map, as they
        # are made once per scan; ragged sizes, volume longer than the scanner
        _case("medium_acf", kind="acf", rings=17, crystals=288, radius=310.0, tang=96,
              nx=111, ny=97, nz=45, vx=4.0, vz=4.0),
        # ordinary-Poisson reconstruction of span-3 data with attenuation
        # factors in the model, zero bins skipped, cut radius; ragged sizes
        _case("span3_weighted_osem", kind="osem", rings=21, crystals=320, radius=330.0, tang=101, span=3,
              nx=131, ny=119, nz=43, vx=3.0, vz=2.0, subsets=10, iterations=2, counts=3e6, bias=True, mult=True,
              skip_zero=True, cut=150.0),
        # reproducible sub-iteration (deterministic option) of a mid-sized scanner
        _case("medium_deterministic", kind="subiteration", rings=16, crystals=256, radius=300.0, tang=75,
              nx=96, ny=96, nz=32, vx=4.0, vz=3.0, subsets=8, counts=1e7, deterministic=True),
        # the headline: one sub-iteration of the clinical scanner
        _case("clinical_subiteration", kind="subiteration"),
        # forward projection of the clinical volume onto all 3.28e7 bins
        _case("clinical_forward", kind="forward"),
        # the clinical subsets' sensitivities of the weighted model: all 16
        # subsets backprojected
        _case("clinical_backward", kind="backward"),
        # one of 32 sub-iterations of a long scanner with 1.5 mm voxels
        _case("large_subiteration", kind="subiteration", rings=64, crystals=640, radius=410.0, pitch=3.2,
              tang=163, nx=320, ny=320, nz=128, vx=1.5, vz=1.5, subsets=32, counts=2e9),
        # one gradient of the differentiable projector: 8 phantoms
        _case("clinical_gradient", kind="gradient", nx=128, ny=128, nz=48, frames=8),
        # 16 uneven reconstructions run as one batch
        _case("batch_osem", kind="batch", problems=16, counts=1e6, subsets=0, iterations=3),
    ]


def _scanner_size(rng, most_rings, least=64):
    rings = int(round(math.exp(rng.uniform(math.log(4), math.log(most_rings)))))
    crystals = 4 * int(round(math.exp(rng.uniform(math.log(least / 4), math.log(160)))))
    radius = round(rng.uniform(0.55, 0.85) * crystals + 60.0, 1)
    return rings, crystals, radius


def draw(rng):
    kind = rng.choice(["forward", "acf", "backward", "subiteration", "subiteration", "osem", "gradient", "batch"])
    if kind == "batch":
        return dict(BASE, kind=kind, problems=rng.randint(2, 16), counts=10 ** rng.uniform(5, 7), subsets=0,
                    iterations=rng.randint(1, 3))
    while True:
        c = dict(BASE, kind=kind)
        rings, crystals, radius = _scanner_size(rng, 64 if kind == "subiteration" else 32)
        c.update(rings=rings, crystals=crystals, radius=radius, pitch=rng.choice([2.0, 3.2, 4.0, 5.0]))
        c["span"] = rng.choice([1, 1, 3]) if rings >= 8 else 1
        c["vx"] = rng.choice([1.5, 2.0, 2.5, 3.0, 4.0])
        c["vz"] = rng.choice([1.5, 2.0, 3.0, 4.0])
        # transaxial field of 0.4 to 0.75 of the diameter; the volume covers
        # the scanner axially, a little more or less
        c["nx"] = max(16, min(320, int(rng.uniform(0.4, 0.75) * 2 * radius / c["vx"])))
        c["ny"] = max(16, c["nx"] - rng.randint(0, 9))
        c["nz"] = max(4, min(128, int(rng.uniform(0.8, 1.5) * rings * c["pitch"] / c["vz"])))
        fov = min(0.45 * c["nx"] * c["vx"], 0.7 * radius)
        c["tang"] = workloads.n_tang_for_fov(crystals, radius, fov) - rng.randint(0, 1)
        views = crystals // 2
        if kind == "gradient":
            c["frames"] = rng.randint(1, 8)
            c["dtype"] = "float64" if c["frames"] < 3 and rng.random() < 0.4 else "float32"
        if kind in ("subiteration", "osem", "backward"):
            c["subsets"] = rng.choice([d for d in range(1, 33) if views % d == 0 and d >= min(4, views)] or [1])
            c["bias"] = rng.random() < 0.5 and kind != "backward"
            c["skip_zero"] = rng.random() < 0.3
        if kind == "osem":
            c["iterations"] = rng.randint(1, 3)
            c["mult"] = rng.random() < 0.4
            c["cut"] = round(0.5 * c["nx"] * c["vx"], 1) if rng.random() < 0.3 else 0.0
        if kind == "subiteration" and rng.random() < 0.15:
            c["deterministic"] = True
        n = _n_bins(c)
        c["counts"] = float(10 ** rng.uniform(-1.5, 1.2) * n)
        if work(c)["flops"] < (4e9 if c["deterministic"] else 4e10) and n * c["frames"] < 4e8:
            return c


# ------------------------------------------------------------- geometry

def _specs(c):
    n_seg = 2 * c["rings"] - 1
    if c["span"] > 1:
        n_seg = (2 * c["rings"] - 1) // c["span"]
        n_seg -= 1 - n_seg % 2
    scanner = ScannerSpec.ring(c["rings"], c["crystals"], c["radius"], c["pitch"])
    proj = ProjSpec(c["rings"], c["crystals"], n_seg, c["tang"], c["span"])
    vol = VolSpec.centred((c["nx"], c["ny"], c["nz"]), (c["vx"], c["vx"], c["vz"]))
    return scanner, proj, vol


def _exact_voxels(c):
    # voxel extents that are not whole mm need the exact geometry
    return any(v != int(v) for v in (c["vx"], c["vz"]))


def _n_axial(c):
    _, proj, _ = _specs(c)
    so = (proj.n_segments - 1) // 2
    out = []
    for s in range(-so, so + 1):
        a = abs(s)
        if c["span"] == 1:
            out.append(c["rings"] - a)
        else:
            out.append(2 * c["rings"] - 1 - (c["span"] + 1 if a >= 1 else 0) - (2 * c["span"] * (a - 1) if a >= 2 else 0))
    return out


def _n_bins(c):
    return sum(_n_axial(c)) * (c["crystals"] // 2) * c["tang"]


def _planes(c):
    """The end slices (a1, a2) of every (segment, axial) row, in file order."""
    nax = _n_axial(c)
    so = (len(nax) - 1) // 2
    span, h = c["span"], (c["span"] - 1) // 2
    rows = []
    for k, n in enumerate(nax):
        seg = k - so
        for ax in range(n):
            if span == 1:
                a1, a2 = (2 * ax, 2 * ax) if seg == 0 else (2 * (ax + seg), 2 * ax) if seg > 0 else (2 * ax, 2 * (ax - seg))
            elif seg == 0:
                a1 = a2 = ax
            else:
                mid, inv = abs(seg) * span, n - ax - 1
                smax = 2 * c["rings"] - 2
                if ax < h:
                    r = 2 * (mid - h + ax)
                    a1, a2 = (r, 0) if seg > 0 else (0, r)
                elif inv < h:
                    r = 2 * (mid - h + inv)
                    a1, a2 = (smax, smax - r) if seg > 0 else (smax - r, smax)
                else:
                    a = ax - h
                    a1, a2 = (2 * mid + a, a) if seg > 0 else (a, 2 * mid + a)
            rows.append((k, a1, a2))
    return nax, rows


def _ends(c, views, device):
    """Crystal centres [n, 6] of the bins of the given views, in FIR's order
    (segment, view, axial, tangential), in 64 bits."""
    nax, rows = _planes(c)
    n, nv, nt = c["crystals"], c["crystals"] // 2, c["tang"]
    ang = torch.arange(n, dtype=torch.float64, device=device) * (2 * math.pi / n)
    cx, cy = c["radius"] * torch.cos(ang), c["radius"] * torch.sin(ang)
    ringz = -((c["rings"] - 1) * c["pitch"]) / 2.0 + c["pitch"] * np.arange(c["rings"], dtype=np.float64)
    k = np.arange(2 * c["rings"] - 1)
    z = torch.from_numpy(np.where(k % 2 == 0, ringz[k // 2], (ringz[k // 2] + ringz[(k + 1) // 2]) / 2.0)).to(device)
    t = torch.arange(nt, device=device) - nt // 2
    shift = torch.div(torch.where(t >= 0, t, t - 1), 2, rounding_mode="trunc")
    v = torch.as_tensor(views, device=device)[:, None]
    c1 = (v + shift + (t.abs() & 1)) % n
    c2 = (v + nv - shift) % n
    flat = torch.stack([cx[c1], cy[c1], cx[c2], cy[c2]], -1)  # [views, tang, 4]
    at = 0
    for m in nax:
        r = rows[at:at + m]
        at += m
        z1 = z[torch.tensor([x[1] for x in r], device=device)]
        z2 = z[torch.tensor([x[2] for x in r], device=device)]
        full = flat[:, None].expand(-1, m, -1, -1)
        za = z1[None, :, None].expand(full.shape[:3])
        zb = z2[None, :, None].expand(full.shape[:3])
        yield torch.stack([full[..., 0], full[..., 1], za, full[..., 2], full[..., 3], zb], -1).reshape(-1, 6)


def _bins_of(c, views, device):
    """Flat bin indices of _ends' rows."""
    nax = _n_axial(c)
    nv, nt = c["crystals"] // 2, c["tang"]
    base = 0
    v = torch.as_tensor(views, device=device)
    for m in nax:
        yield (base + v[:, None] * (m * nt) + torch.arange(m * nt, device=device)[None]).reshape(-1)
        base += m * nv * nt


# ------------------------------------------------------------- inputs

def _phantom(c, gen, device, frames):
    """Activity [frames, nz, ny, nx]: an elliptical body with hot and cold
    ellipsoids, with the grain of an estimate between iterations."""
    _, _, vol = _specs(c)
    x, y, z = (torch.from_numpy(a).to(device, torch.float32) for a in vol.voxel_centres())
    Z, Y, X = z[:, None, None], y[None, :, None], x[None, None, :]
    hx, hz = 0.5 * c["nx"] * c["vx"], 0.5 * c["nz"] * c["vz"]
    a, b = 0.8 * hx, 0.6 * hx
    out = torch.zeros((frames, c["nz"], c["ny"], c["nx"]), device=device)
    u = torch.rand((frames, 8, 8), generator=gen, device=device).cpu().numpy()
    body = ((X / a) ** 2 + (Y / b) ** 2 <= 1).expand(out.shape[1:])
    for f in range(frames):
        img = body.float()
        for q in u[f]:
            e = ((X - (q[0] - .5) * 1.4 * a) / (0.05 + 0.3 * q[1]) / a) ** 2 + \
                ((Y - (q[2] - .5) * 1.4 * b) / (0.05 + 0.3 * q[3]) / a) ** 2 + \
                ((Z - (q[4] - .5) * 1.6 * hz) / (0.1 + 0.7 * q[5]) / max(hz, 1.0)) ** 2 <= 1
            img = torch.where(e & body, torch.tensor(0.2 + 5.0 * float(q[6]), device=device), img)
        out[f] = img
    return out * (0.7 + 0.6 * torch.rand(out.shape, generator=gen, device=device))


def _chords(c, device):
    """Chord of every bin's line through the elliptical body (mm), float32 in
    file order, and its in-plane distance from the hot insert's centre."""
    hx = 0.5 * c["nx"] * c["vx"]
    a, b = 0.8 * hx, 0.6 * hx
    n, nv, nt = c["crystals"], c["crystals"] // 2, c["tang"]
    one = dict(c, rings=1, span=1)
    e = torch.cat(list(_ends(one, np.arange(nv), device)))  # [nv * nt, 6]
    dx, dy = e[:, 3] - e[:, 0], e[:, 4] - e[:, 1]
    A = (dx / a) ** 2 + (dy / b) ** 2
    B = 2 * (e[:, 0] * dx / a ** 2 + e[:, 1] * dy / b ** 2)
    C = (e[:, 0] / a) ** 2 + (e[:, 1] / b) ** 2 - 1
    ln = torch.sqrt(torch.clamp(B * B - 4 * A * C, min=0)) / A * torch.sqrt(dx * dx + dy * dy)
    ln = ln.float().reshape(nv, 1, nt)
    return torch.cat([ln.expand(nv, m, nt).reshape(-1) for m in _n_axial(c)])


def _measured(c, gen, device, frames=1):
    """Counts of the attenuated body (Poisson), precorrected unless the model
    is weighted, and the attenuation factors exp(-mu chord)."""
    ln = _chords(c, device)
    atten = torch.exp(-0.0096 * ln)
    mean = ln * atten * (0.8 + 0.4 * torch.rand(ln.shape, generator=gen, device=device))
    mean *= float(c["counts"] / max(float(mean.sum(dtype=torch.float64)), 1e-30))
    ys = []
    for _ in range(frames):
        ys.append(torch.poisson(mean, generator=gen))
        if not c["mult"] and c["kind"] != "gradient":
            ys[-1] /= atten
    return (ys[0] if frames == 1 else torch.stack(ys)), atten


def _params(c):
    f = c["fwhm"] if c["kind"] in ("osem", "subiteration", "batch") else 0.0
    return OSEMParams(n_iterations=c["iterations"], n_subsets=c["subsets"], cut_radius=c["cut"],
                      convolution_interval=1 if f > 0 else 0, fwhm_xyz=[f, f, f])


def _context(c, scanner):
    ctx = capi.Context(scanner)
    if _exact_voxels(c):
        ctx.set_option(capi.FIR_OPT_GEOMETRY, capi.FIR_GEOMETRY_EXACT)
    if c["skip_zero"]:
        ctx.set_option(capi.FIR_OPT_SKIP_ZERO_BINS, 1)
    if c["deterministic"]:
        ctx.set_option(capi.FIR_OPT_BACKPROJ_MODE, capi.FIR_BACKPROJ_DETERMINISTIC)
    return ctx


def _inputs(case, seed):
    """The input arrays of a case, from the seed alone (this file's code)."""
    c = dict(BASE)
    c.update(case)
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    d = {}
    kind = c["kind"]
    if kind in ("forward", "acf"):
        d["img"] = _phantom(c, gen, dev, 1)[0] * (0.0096 if kind == "acf" else 1.0)
    elif kind == "backward":
        d["y"], atten = _measured(c, gen, dev)
        if not c["skip_zero"]:
            d["y"] = atten * (0.5 + torch.rand(atten.shape, generator=gen, device=dev))
    elif kind in ("subiteration", "osem"):
        d["y"], atten = _measured(c, gen, dev)
        d["mult"] = atten if c["mult"] else None
        d["bias"] = None
        if c["bias"]:
            r = 0.2 * float(d["y"].mean()) + 1e-3
            d["bias"] = r * (0.5 + torch.rand(d["y"].shape, generator=gen, device=dev))
        d["img"] = torch.ones((c["nz"], c["ny"], c["nx"]), device=dev)
        if kind == "subiteration":
            d["img"] = _phantom(c, gen, dev, 1)[0] + 0.05
    elif kind == "gradient":
        dt = getattr(torch, c["dtype"])
        x = _phantom(c, gen, dev, c["frames"]) + 0.05
        y, atten = _measured(c, gen, dev, c["frames"])
        y = y.reshape(c["frames"], -1)
        if c["counts"] > 0:
            x *= float(c["counts"] / _n_bins(c)) / 50.0
        d.update(x=x.to(dt), y=y.to(dt), atten=atten.to(dt)[None], bias=0.05 * float(y.mean()) + 1e-3)
    return c, d


def prepare(case, seed):
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    c, d = _inputs(case, seed)
    scanner, proj, vol = _specs(c)
    s = dict(c=c, proj=proj, vol=vol, prm=_params(c), **d)
    dev = torch.device("cuda")
    if c["kind"] == "gradient":
        geo = capi.FIR_GEOMETRY_EXACT if _exact_voxels(c) else None
        s["op"] = autograd.SiddonProjector(scanner, proj, vol, geometry=geo)
        return s
    s["ctx"] = ctx = _context(c, scanner)
    nb = _n_bins(c)
    if c["kind"] in ("forward", "acf"):
        s["out"] = torch.empty(nb, device=dev)
    elif c["kind"] == "backward":
        s["out"] = torch.empty((c["subsets"],) + vol.shape_zyx, device=dev)
    else:
        # sensitivity of the subsets the case uses: A_s^T m
        s["sens"] = torch.empty((c["subsets"],) + vol.shape_zyx, device=dev)
        if c["mult"]:
            ctx.backward(proj, s["mult"], vol, s["sens"], c["subsets"])
        else:
            with capi.Context(scanner) as plain:
                if _exact_voxels(c):
                    plain.set_option(capi.FIR_OPT_GEOMETRY, capi.FIR_GEOMETRY_EXACT)
                plain.sensitivity(proj, vol, s["sens"], c["subsets"])
                plain.synchronize()
        if c["kind"] == "subiteration":
            s["sens"] = s["sens"][c["subsets"] // 3].clone()
        s["work"] = torch.empty_like(s["img"])
    ctx.synchronize()
    return s


def _batch_of(case):
    return workloads.batch_problems(case["problems"])


def _problem_case(case, w):
    """The case fields of one problem of a batch."""
    return dict(BASE, kind="osem", rings=w.proj.n_rings, crystals=w.proj.n_crystals_per_ring,
                radius=w.scanner.rsector_inner_radius, pitch=4.0, tang=w.proj.n_tang_coords, nx=w.vol.size[0],
                ny=w.vol.size[1], nz=w.vol.size[2], vx=w.vol.voxel[0], vz=w.vol.voxel[2], subsets=w.osem.n_subsets,
                iterations=case["iterations"], counts=case["counts"])


def _prepare_batch(case, seed):
    ws = _batch_of(case)
    ctx = capi.Context(ws[0].scanner)
    cs = [_problem_case(case, w) for w in ws]
    batch = capi.Batch(ctx, [(w.scanner, w.proj, w.vol, _params(c)) for w, c in zip(ws, cs)])
    start = []
    for k, (w, c) in enumerate(zip(ws, cs)):
        c, d = _inputs(c, seed + 7919 * (k + 1))
        ctx.set_scanner(w.scanner)
        sens = torch.empty((c["subsets"],) + w.vol.shape_zyx, device="cuda")
        ctx.sensitivity(w.proj, w.vol, sens, c["subsets"])
        ctx.synchronize()
        batch.set_data(k, d["y"], sens)
        start.append(d["img"])
    torch.cuda.synchronize()
    return dict(c=dict(BASE, **{k: v for k, v in case.items()}), ctx=ctx, batch=batch, start=start,
                out=[torch.empty_like(x) for x in start])


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "batch":
        # a reconstruction of new images with the batch a program keeps
        for k, x in enumerate(s["start"]):
            s["batch"].set_image(k, x)
        s["batch"].osem()
        for k, x in enumerate(s["out"]):
            s["batch"].get_image(k, x)
        return s["out"]
    if kind == "gradient":
        x = s["x"].detach().requires_grad_(True)
        loss = autograd.penalized_nll(x, s["y"], s["op"], 0.01, s["atten"], s["bias"])
        loss.backward()
        return [loss.detach(), x.grad]
    ctx, proj, vol = s["ctx"], s["proj"], s["vol"]
    if kind == "forward":
        ctx.forward(vol, s["img"], proj, s["out"])
        return s["out"]
    if kind == "acf":
        ctx.forward_exp(vol, s["img"], proj, s["out"])
        return s["out"]
    if kind == "backward":
        ctx.backward(proj, s["y"], vol, s["out"], c["subsets"])
        return s["out"]
    s["work"].copy_(s["img"])
    if kind == "subiteration":
        ctx.osem_subiteration(proj, s["y"], vol, s["work"], s["sens"], s["prm"], c["subsets"] // 3, 1, bias=s["bias"])
    else:
        ctx.osem(proj, s["y"], vol, s["work"], s["sens"], s["prm"], bias=s["bias"], mult=s["mult"])
    return s["work"]


# ------------------------------------------------------------- work

def _mean_steps(c):
    """Mean number of voxels a line of response crosses (4096 random lines)."""
    r = np.random.RandomState(3)
    n, nv, nt, m = c["crystals"], c["crystals"] // 2, c["tang"], 4096
    rows = _planes(c)[1]
    pick = r.randint(0, len(rows), m)
    a = np.array(rows)[pick]
    v, t = r.randint(0, nv, m), r.randint(0, nt, m) - nt // 2
    shift = np.where(t >= 0, t, t - 1) / 2
    shift = np.trunc(shift).astype(int)
    c1, c2 = (v + shift + (np.abs(t) & 1)) % n, (v + nv - shift) % n
    half = (c["rings"] - 1) * c["pitch"] / 2
    p = [np.stack([c["radius"] * np.cos(2 * np.pi * k / n), c["radius"] * np.sin(2 * np.pi * k / n),
                   a[:, j] * c["pitch"] / 2 - half]) for k, j in ((c1, 1), (c2, 2))]
    d = p[1] - p[0]
    d = np.where(np.abs(d) < 1e-9, 1e-9, d)
    box = np.array([c["nx"] * c["vx"], c["ny"] * c["vx"], c["nz"] * c["vz"]])[:, None] / 2
    lo, hi = np.minimum((-box - p[0]) / d, (box - p[0]) / d), np.maximum((-box - p[0]) / d, (box - p[0]) / d)
    f = np.clip(np.minimum(hi.min(0), 1) - np.maximum(lo.max(0), 0), 0, None)
    ext = np.array([c["vx"], c["vx"], c["vz"]])[:, None]
    return float(((np.abs(d) * f / ext).sum(0) + (f > 0)).mean())


def work(case):
    """Bytes: every input read and every output written once.  Operations:
    per voxel of a path and traversal four (the length's difference and
    product, the product with the value, the sum)."""
    if case["kind"] == "batch":
        ws = [work(_problem_case(case, w)) for w in _batch_of(case)]
        return {k: float(sum(x[k] for x in ws)) for k in ("bytes", "flops")}
    c = dict(BASE)
    c.update(case)
    nb, nvox = _n_bins(c), c["nx"] * c["ny"] * c["nz"]
    steps = _mean_steps(c)
    es = 8 if c["dtype"] == "float64" else 4
    arrays = 1 + c["bias"] + c["mult"]
    kind = c["kind"]
    if kind in ("forward", "acf"):
        return {"bytes": 4.0 * (nb + nvox), "flops": 4.0 * steps * nb}
    if kind == "backward":
        return {"bytes": 4.0 * (nb + nvox * c["subsets"]), "flops": 4.0 * steps * nb}
    if kind == "gradient":
        f = c["frames"]
        # the measured data and factors, the image and its gradient
        return {"bytes": es * (nb * (f + 1.0) + 2.0 * f * nvox), "flops": 2.0 * steps * nb * (2 + 2 * f)}
    if kind == "subiteration":
        n = nb / c["subsets"]
        return {"bytes": 4.0 * (n * arrays + 3 * nvox), "flops": 8.0 * steps * n}
    return {"bytes": 4.0 * (nb * arrays + nvox * (c["subsets"] + 2.0)), "flops": 8.0 * steps * nb * c["iterations"]}


# ------------------------------------------------------------- 64 bits

def _walk(c, e, visit):
    """FIR's traversal of the lines e [n, 6] in 64 bits, all lines a step at a
    time: visit(lines, voxel, length) for the voxels inside the volume."""
    _, _, vol = _specs(c)
    n = torch.tensor([c["nx"], c["ny"], c["nz"]], device=e.device)
    vox = [c["vx"], c["vx"], c["vz"]]
    low = [vol.offset[0] - vox[0] / 2, vol.offset[1] - vox[1] / 2, vol.offset[2] - c["nz"] * vox[2] / 2]
    d, amin, amax, a, da, ind, step = [], None, None, [], [], [], []
    lo_s, hi_s, first, miss = [], [], [], torch.zeros(len(e), dtype=torch.bool, device=e.device)
    for k in range(3):
        lo = low[k]
        hi = lo + int(n[k]) * vox[k]
        c1, df = e[:, k], e[:, 3 + k] - e[:, k]
        par = ~(df.abs() > EPS)
        miss |= par & ((c1 < lo) | (c1 > hi))
        df = torch.where(par, torch.full_like(df, EPS), df)
        up = (df > 0) & ~par
        s0 = torch.where(up, (lo - c1) / df, (hi - c1) / df)
        s1 = torch.where(up, (hi - c1) / df, (lo - c1) / df)
        lo_s.append(torch.where(par, torch.zeros_like(df), s0))
        hi_s.append(torch.where(par, torch.ones_like(df), s1))
        d.append(df)
        first.append(par)
        step.append(torch.where(up, 1, -1))
    zero, one = torch.zeros_like(d[0]), torch.ones_like(d[0])
    amin = torch.maximum(lo_s[0], torch.maximum(lo_s[1], torch.maximum(lo_s[2], zero)))
    amax = torch.minimum(hi_s[0], torch.minimum(hi_s[1], torch.minimum(hi_s[2], one)))
    d12 = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
    for k in range(3):
        i = torch.trunc((e[:, k] + d[k] * amin - low[k]) / vox[k]).long()
        i = i.clamp(0, int(n[k]) - 1)
        dk = (vox[k] / d[k]).abs()
        al = torch.where(first[k], one, (low[k] + vox[k] * i - e[:, k]) / d[k])
        a.append(torch.where(step[k] > 0, al + dk, al))
        da.append(dk)
        ind.append(i)
    ok = ~miss & (amin < amax)
    at = torch.nonzero(ok).reshape(-1)
    a, da, ind, step = ([x[at] for x in v] for v in (a, da, ind, step))
    prev, end, d12 = amin[at], amax[at], d12[at]
    k = 0
    while len(at):
        nxt = torch.minimum(end, torch.minimum(a[0], torch.minimum(a[1], a[2])))
        inside = prev < end
        for q in range(3):
            inside &= (ind[q] >= 0) & (ind[q] < n[q])
        cell = (ind[2] * c["ny"] + ind[1]) * c["nx"] + ind[0]
        visit(at, torch.where(inside, cell, torch.zeros_like(cell)), torch.where(inside, (nxt - prev) * d12, zero[:1]))
        for q in range(3):
            hit = (a[q] - nxt).abs() < EPS
            a[q] = torch.where(hit, a[q] + da[q], a[q])
            ind[q] = torch.where(hit, ind[q] + step[q], ind[q])
        prev = nxt
        k += 1
        if k % 32 == 0:
            keep = torch.nonzero(prev < end).reshape(-1)
            at, prev, end, d12 = at[keep], prev[keep], end[keep], d12[keep]
            a, da, ind, step = ([x[keep] for x in v] for v in (a, da, ind, step))


_CHUNK = 1 << 21


def _chunks(c, views, device):
    for e, b in zip(_ends(c, views, device), _bins_of(c, views, device)):
        for k in range(0, len(b), _CHUNK):
            yield e[k:k + _CHUNK], b[k:k + _CHUNK]


def _joined(c, views, device):
    """Chunks of about _CHUNK lines across segments."""
    es, bs, n = [], [], 0
    for e, b in _chunks(c, views, device):
        es.append(e)
        bs.append(b)
        n += len(b)
        if n >= _CHUNK:
            yield torch.cat(es), torch.cat(bs)
            es, bs, n = [], [], 0
    if n:
        yield torch.cat(es), torch.cat(bs)


def _project(c, img, e):
    """Line integrals [F, n] of img [F, nvox] along e."""
    out = torch.zeros((len(img), len(e)), dtype=torch.float64, device=e.device)

    def visit(at, cell, ln):
        for f in range(len(img)):
            out[f].index_add_(0, at, ln * img[f][cell])

    _walk(c, e, visit)
    return out


def _scatter(c, acc, vals, e):
    """acc [F, nvox] += backprojection of vals [F, n] along e."""
    def visit(at, cell, ln):
        for f in range(len(acc)):
            acc[f].index_add_(0, cell, ln * vals[f][at])

    _walk(c, e, visit)


def _filter(c, img, fwhm):
    """The separable Gaussian with the edges' weights renormalised."""
    x = img.reshape(c["nz"], c["ny"], c["nx"])
    for axis, vox in ((2, c["vx"]), (1, c["vx"]), (0, c["vz"])):
        sigma = fwhm / 2.3548
        half = (int(6.0 * sigma / vox) + 1) // 2
        n = x.shape[axis]
        num, den = torch.zeros_like(x), torch.zeros(n, dtype=x.dtype, device=x.device)
        for k in range(-half, half + 1):
            w = math.exp(-(k * k * vox * vox) / (2 * sigma * sigma))
            a, b = max(0, -k), min(n, n - k)
            if b > a:
                num.narrow(axis, a, b - a).add_(w * x.narrow(axis, a + k, b - a))
                den[a:b] += w
        shape = [1, 1, 1]
        shape[axis] = n
        x = num / den.reshape(shape)
    return x.reshape(-1)


def _radius(c, device):
    px = c["vx"] * (torch.arange(c["nx"], device=device, dtype=torch.float64) + 0.5 - c["nx"] / 2)
    py = c["vx"] * (torch.arange(c["ny"], device=device, dtype=torch.float64) + 0.5 - c["ny"] / 2)
    r = torch.sqrt(px[None] ** 2 + py[:, None] ** 2)
    return r[None].expand(c["nz"], -1, -1).reshape(-1)


def _exact_osem(c, d):
    dev = d["y"].device
    img = d["img"].double().reshape(-1)
    r = _radius(c, dev)
    views = np.arange(c["crystals"] // 2)
    if c["kind"] == "osem" and c["cut"] > 0:
        img = torch.where(r > c["cut"], torch.zeros_like(img), img)
    order = [c["subsets"] // 3] if c["kind"] == "subiteration" else list(range(c["subsets"])) * c["iterations"]
    sens = {}
    for sub in order:
        bp = torch.zeros((2, img.numel()), dtype=torch.float64, device=dev)
        for e, b in _joined(c, views[views % c["subsets"] == sub], dev):
            y = d["y"][b].double()
            m = d["mult"][b].double() if d["mult"] is not None else torch.ones_like(y)
            line = _project(c, img[None], e)[0] * m
            if d["bias"] is not None:
                line = line + d["bias"][b].double()
            q = torch.where(line > EPS, y / line * m, torch.zeros_like(y))
            _scatter(c, bp if sub not in sens else bp[:1], torch.stack([q, m]), e)
        if sub not in sens:
            sens[sub] = bp[1]
        s = sens[sub]
        zero = torch.zeros_like(img)
        q = torch.where((bp[0] > EPS) & (s > EPS), bp[0] / s, zero)
        img = torch.where((img > EPS) & (q > EPS), img * q, zero)
        old = img
        img = _filter(c, img, c["fwhm"])
        if c["cut"] > 0:
            img = torch.where(r >= c["cut"] - 5.0 * c["fwhm"], old, img)
            img = torch.where(r > c["cut"], zero, img)
    return img.reshape(c["nz"], c["ny"], c["nx"])


def _exact_gradient(c, d):
    dev = d["y"].device
    x = d["x"].double()
    flat = x.reshape(c["frames"], -1)
    grad = torch.zeros_like(flat)
    loss = torch.zeros((), dtype=torch.float64, device=dev)
    for e, b in _joined(c, np.arange(c["crystals"] // 2), dev):
        y, m = d["y"][:, b].double(), d["atten"][0, b].double()
        mean = _project(c, flat, e) * m + d["bias"]
        loss += (mean - torch.xlogy(y, mean)).sum()
        _scatter(c, grad, m * (1 - y / mean), e)
    with torch.enable_grad():
        xg = x.detach().requires_grad_(True)
        pen = torch.zeros((), dtype=torch.float64, device=dev)
        nz, ny, nx = x.shape[-3:]
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    if (dz, dy, dx) > (0, 0, 0):
                        p = xg[:, max(dz, 0):nz + min(dz, 0), max(dy, 0):ny + min(dy, 0), max(dx, 0):nx + min(dx, 0)]
                        q = xg[:, max(-dz, 0):nz + min(-dz, 0), max(-dy, 0):ny + min(-dy, 0), max(-dx, 0):nx + min(-dx, 0)]
                        pen = pen + ((p - q) ** 2).sum() / math.sqrt(dz * dz + dy * dy + dx * dx)
        pen = 0.5 * 0.01 * pen
        pen.backward()
    return [loss + pen.detach(), grad.reshape(x.shape) + xg.grad]


def exact(case, seed):
    if case["kind"] == "batch":
        return None
    c, d = _inputs(case, seed)
    total = work(c)["flops"] / 4 * (2 if c["kind"] == "osem" else 1)
    if total > 1.5e11:
        return None
    dev = torch.device("cuda")
    views = np.arange(c["crystals"] // 2)
    with torch.no_grad():
        if c["kind"] in ("forward", "acf"):
            out = torch.zeros(_n_bins(c), dtype=torch.float64, device=dev)
            img = d["img"].double().reshape(1, -1)
            for e, b in _joined(c, views, dev):
                out[b] = _project(c, img, e)[0]
            return torch.where(out > EPS, torch.exp(out), torch.ones_like(out)) if c["kind"] == "acf" else out
        if c["kind"] == "backward":
            out = torch.zeros((c["subsets"], c["nx"] * c["ny"] * c["nz"]), dtype=torch.float64, device=dev)
            for sub in range(c["subsets"]):
                for e, b in _joined(c, views[views % c["subsets"] == sub], dev):
                    _scatter(c, out[sub:sub + 1], d["y"][b].double()[None], e)
            return out.reshape(c["subsets"], c["nz"], c["ny"], c["nx"])
        if c["kind"] == "gradient":
            return _exact_gradient(c, d)
        return _exact_osem(c, d)
