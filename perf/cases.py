"""The calls that users of nefct_b200 make, as cases with inputs, one pass and a float64 value.

Kinds of case (field ``kind``); sizes come from the repository's own workloads (the 64^3, 256^3,
512^3, batched and motion scans of bench.py, README.md and the tests) or are ordinary scanner
sizes around them:

* ``pair``    one differentiable projection: ops.project and its vector-Jacobian product, i.e.
              forward projector and exact transpose (training, gradient descent, unrolled loops);
* ``fdk``     a whole FDK reconstruction (weighting, ramp filter, backprojection);
* ``lor``     the line-of-response pair over a PET-like line list;
* ``motion``  4-D: warp the reference volume per phase, project it, gradients of volume and fields;
* ``dd``      the distance-driven pair through autograd;
* ``batch``   many small uneven problems through one batch plan;
* ``solve``   a whole iterative reconstruction (SIRT or conjugate gradients).

Everything is float32, as users run it; the float64 builds of the operators serve checks only.
"""
import math

import numpy as np
import torch

import nefct_b200 as nb
from nefct_b200 import _lib, ops, recon
from nefct_b200.batch import BatchProjector, batch_project

DEV = "cuda"


# ---------------- cases ----------------

def _pair(name, shape, voxel, nv, na, nb_, pixel, si, sd, det="flat", pitch=0.0, line=False, deterministic=False):
    c = dict(kind="pair", nx=shape[0], ny=shape[1], nz=shape[2], vx=voxel[0], vy=voxel[1], vz=voxel[2], nv=nv, na=na,
             nb=nb_, px=pixel, si=si, sd=sd, det=det, pitch=pitch, line=line, deterministic=deterministic)
    return dict(c, name=name) if name else c


def _fdk(name, shape, voxel, nv, na, nb_, pixel, si, sd, window="ram-lak", short=False):
    c = dict(kind="fdk", nx=shape[0], ny=shape[1], nz=shape[2], vx=voxel, vy=voxel, vz=voxel, nv=nv, na=na, nb=nb_,
             px=pixel, si=si, sd=sd, window=window, short=short)
    return dict(c, name=name) if name else c


def _lor(name, shape, lines, ordered):
    c = dict(kind="lor", nx=shape[0], ny=shape[1], nz=shape[2], lines=lines, ordered=ordered)
    return dict(c, name=name) if name else c


def _motion(name, n, phases, per, na, nb_, pixel):
    c = dict(kind="motion", n=n, phases=phases, per=per, na=na, nb=nb_, px=pixel, si=600.0, sd=1200.0)
    return dict(c, name=name) if name else c


def _dd(name, shape, nv, na, nb_, pixel, weight):
    c = dict(kind="dd", nx=shape[0], ny=shape[1], nz=shape[2], nv=nv, na=na, nb=nb_, px=pixel, sad=600.0, sid=1200.0,
             weight=weight)
    return dict(c, name=name) if name else c


def _batch(name, problems, lo, hi, vlo, vhi, dlo, dhi, pick):
    c = dict(kind="batch", problems=problems, lo=lo, hi=hi, vlo=vlo, vhi=vhi, dlo=dlo, dhi=dhi, pick=pick)
    return dict(c, name=name) if name else c


def _solve(name, solver, n, nv, na, nb_, pixel, iters):
    c = dict(kind="solve", solver=solver, n=n, nv=nv, na=na, nb=nb_, px=pixel, si=500.0, sd=1000.0, iters=iters)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small scan in a training loop: launches and latency count
        _pair("pair_64cube", (64, 64, 64), (2.0, 2.0, 2.0), 90, 128, 96, 2.0, 500.0, 1000.0),
        # the ordinary scanner: 256^3, 360 views of 512 x 384
        _pair("pair_256cube", (256, 256, 256), (1.0, 1.0, 1.0), 360, 512, 384, 1.2, 600.0, 1200.0),
        # the largest scan on one GPU: 512^3, 720 views of 1024 x 768
        _pair("pair_512cube", (512, 512, 512), (1.0, 1.0, 1.0), 720, 1024, 768, 1.0, 700.0, 1400.0),
        # a helical scan on a cylindrical detector, slices thicker than the pixels, nothing a multiple of 32
        _pair("pair_helical_cyl", (211, 203, 83), (1.0, 1.0, 2.5), 237, 443, 77, 1.3, 570.0, 1040.0, det="cyl",
              pitch=60.0, line=True),
        # reproducible training: the bitwise reproducible transpose
        _pair("pair_deterministic", (160, 160, 128), (1.0, 1.0, 1.0), 96, 320, 256, 1.2, 600.0, 1200.0,
              deterministic=True),
        # FDK on the ordinary scanner
        _fdk("fdk_256cube", (256, 256, 256), 1.0, 360, 512, 384, 1.2, 600.0, 1200.0),
        # FDK of a short scan with Parker weights, odd sizes
        _fdk("fdk_short_scan", (187, 193, 121), 1.2, 211, 389, 283, 1.3, 600.0, 1200.0, window="hann", short=True),
        # PET: a list of 4 Mi lines in walk order
        _lor("lor_4M_ordered", (256, 256, 256), 4 << 20, True),
        # motion-compensated 4-D step with image and field gradients
        _motion("motion_192cube", 192, 4, 40, 400, 300, 1.2),
        # the distance-driven pair
        _dd("dd_256cube", (256, 256, 256), 48, 512, 384, 1.2, False),
        # a minibatch of small uneven reconstructions in one plan
        _batch("batch_28_small", 28, 16, 64, 8, 64, 24, 128, 44),
        # a small iterative reconstruction, ten SIRT iterations
        _solve("sirt_96cube", "sirt", 96, 120, 160, 130, 1.3, 10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "pair", "pair", "pair", "fdk", "lor", "motion", "dd", "batch", "solve"])
    if kind in ("pair", "fdk", "dd"):
        n = _log_int(rng, 32, 256)
        shape = (n, max(8, int(n * rng.uniform(0.8, 1.2))), max(8, int(n * rng.uniform(0.3, 1.1))))
        # the detector covers between most and all of the magnified volume
        fine = rng.uniform(0.9, 1.9)                    # pixels per voxel at the axis
        cover = rng.uniform(0.8, 1.3)
        na, rows = max(16, int(n * fine * cover)), max(8, int(shape[2] * fine * cover))
    if kind == "pair":
        v = rng.choice([0.5, 1.0, 2.0])
        vz = v * rng.choice([1.0, 1.0, 1.0, 1.6, 2.5])
        mag = rng.uniform(1.5, 2.0)
        si = max(400.0, 2.2 * v * n) * rng.uniform(1.0, 1.3)
        det = rng.choice(["flat", "flat", "flat", "cyl"])
        return _pair(None, shape, (v, v, vz), _log_int(rng, 20, 400), na, rows, round(v * mag / fine, 3), round(si, 1),
                     round(si * mag, 1), det=det, pitch=round(rng.choice([0.0, 0.0, 0.5]) * vz * shape[2], 2),
                     line=rng.random() < 0.5, deterministic=rng.random() < 0.15)
    if kind == "fdk":
        v = rng.choice([0.5, 1.0, 1.2])
        si = round(max(400.0, 2.2 * v * n) * rng.uniform(1.0, 1.3), 1)
        return _fdk(None, shape, v, _log_int(rng, 60, 400), na, rows, round(v * 2.0 / fine, 3), si, 2 * si,
                    window=rng.choice(["ram-lak", "shepp-logan", "cosine", "hamming", "hann"]), short=rng.random() < 0.3)
    if kind == "dd":
        return _dd(None, shape, _log_int(rng, 12, 60), na, rows, round(2.0 / fine, 3), rng.random() < 0.5)
    if kind == "lor":
        n = _log_int(rng, 64, 300)
        return _lor(None, (n, n + rng.randint(-9, 9), max(16, int(n * rng.uniform(0.4, 1.0)))),
                    _log_int(rng, 20_000, 6_000_000), rng.random() < 0.7)
    if kind == "motion":
        n = _log_int(rng, 48, 192)
        return _motion(None, n, rng.randint(2, 4), _log_int(rng, 10, 40), int(n * 2.05), int(n * 1.5), 1.2)
    if kind == "batch":
        return _batch(None, rng.randint(4, 30), 16, rng.randint(40, 72), 8, rng.randint(24, 72), 24,
                      rng.randint(64, 160), rng.randint(0, 1 << 20))
    n = _log_int(rng, 32, 144)
    return _solve(None, rng.choice(["sirt", "sirt", "cg"]), n, _log_int(rng, 30, 160), int(n * 1.7), int(n * 1.3), 1.3,
                  rng.randint(2, 8))


# ---------------- inputs ----------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _phantom(shape, seed, ellipsoids=8):
    """Sum of random ellipsoids in a body ellipsoid, [nz, ny, nx] float32 (an attenuation image)."""
    nz, ny, nx = shape
    rng = np.random.default_rng(seed)
    z = torch.linspace(-1, 1, nz, device=DEV).view(-1, 1, 1)
    y = torch.linspace(-1, 1, ny, device=DEV).view(1, -1, 1)
    x = torch.linspace(-1, 1, nx, device=DEV).view(1, 1, -1)
    vol = 0.2 * ((x / 0.9) ** 2 + (y / 0.85) ** 2 + (z / 0.95) ** 2 <= 1).float()
    for _ in range(ellipsoids):
        c, a = rng.uniform(-0.55, 0.55, 3), rng.uniform(0.05, 0.35, 3)
        inside = ((x - c[0]) / a[0]) ** 2 + ((y - c[1]) / a[1]) ** 2 + ((z - c[2]) / a[2]) ** 2 <= 1
        vol += float(rng.uniform(0.1, 1.0)) * inside
    return vol


def _angles(c):
    if c.get("short"):
        fan = 2 * math.degrees(math.atan(c["na"] * c["px"] / 2 / c["sd"]))
        return np.deg2rad((np.arange(c["nv"]) / c["nv"]) * (180.0 + fan) - fan / 2).astype(np.float32)
    turns = 2.0 if c.get("pitch") else 1.0
    return np.linspace(0, 2 * np.pi * turns, c["nv"], endpoint=False).astype(np.float32)


def _cone(c):
    """ops.ConeBeam arguments of a cone-beam case."""
    n = c.get("n")
    shape = (n, n, n) if n else (c["nx"], c["ny"], c["nz"])
    vox = (1.0, 1.0, 1.0) if n else (c["vx"], c["vy"], c["vz"])
    cyl = c.get("det") == "cyl"
    off = None
    if c.get("pitch"):
        off = (np.linspace(-0.5, 0.5, c["nv"]) * c["pitch"]).astype(np.float32)
    return dict(shape=shape, angles=_angles(c), src_iso=c["si"], src_det=c["sd"], na=c["na"],
                da=c["px"] / c["sd"] if cyl else c["px"], nb=c["nb"], db=c["px"],
                size=tuple(s * v for s, v in zip(shape, vox)), det_kind="cyl" if cyl else "flat", z_offsets=off)


def _flags(c):
    return (_lib.LINE_INTEGRAL if c["line"] else _lib.REF_FORWARD) | (_lib.DETERMINISTIC if c["deterministic"] else 0)


def _ring_lines(c, seed):
    """Random lines between points of a ring around the grid, [6, n] (a PET line list)."""
    r, half = 0.62 * max(c["nx"], c["ny"]), 0.4 * c["nz"]
    u = torch.rand((4, c["lines"]), device=DEV, generator=_gen(seed))
    p1, p2 = 2 * math.pi * u[0], 2 * math.pi * u[1]
    return torch.stack([r * p1.cos(), r * p1.sin(), (2 * u[2] - 1) * half, r * p2.cos(), r * p2.sin(),
                        (2 * u[3] - 1) * half]).contiguous()


def _motion_cones(c):
    ang = np.linspace(0, 2 * np.pi, c["phases"] * c["per"], endpoint=False).astype(np.float32)
    one = dict(c, nv=c["per"])
    return [dict(_cone(one), angles=ang[p::c["phases"]]) for p in range(c["phases"])]


def _fields(c, seed):
    """Smooth displacement fields of up to 5 voxels per phase, three [n, n, n] components each."""
    n, rng = c["n"], np.random.default_rng(seed)
    t = torch.linspace(0, 1, n, device=DEV)
    z, y, x = t.view(-1, 1, 1), t.view(1, -1, 1), t.view(1, 1, -1)
    amp = 5.0 * n / 256
    out = []
    for _ in range(c["phases"]):
        comps = []
        for _ in range(3):
            f = torch.zeros((n, n, n), device=DEV)
            for _ in range(4):
                kx, ky, kz = rng.uniform(0.3, 2.0, 3)
                f += 0.25 * amp * torch.sin(2 * math.pi * (kx * x + ky * y + kz * z) + float(rng.uniform(0, 6.28)))
            comps.append(f)
        out.append(comps)
    return out


def _batch_cones(c):
    rng = np.random.default_rng(c["pick"])
    out = []
    for _ in range(c["problems"]):
        n = int(round(math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"])))))
        nv = int(rng.integers(c["vlo"], c["vhi"] + 1))
        rows, cols = (int(v) for v in rng.integers(c["dlo"], c["dhi"] + 1, 2))
        si = float(rng.uniform(400, 700))
        sd = si * float(rng.uniform(1.5, 2.0))
        pixel = (sd / si) * n / cols
        out.append(dict(shape=(n, n, n), angles=np.linspace(0, 2 * np.pi, nv, endpoint=False).astype(np.float32),
                        src_iso=si, src_det=sd, na=cols, da=pixel, nb=rows, db=pixel, size=(float(n),) * 3,
                        det_kind="flat", z_offsets=None))
    return out


def _sino_shape(k):
    return (len(k["angles"]), k["nb"], k["na"])


def _vol_shape(k):
    return tuple(reversed(k["shape"]))


def _soft_sino(shape, seed):
    """A projection-like sinogram: smooth across the detector, strictly positive, a little noise."""
    nv, rows, cols = shape
    u = torch.linspace(-1, 1, cols, device=DEV).view(1, 1, -1)
    v = torch.linspace(-1, 1, rows, device=DEV).view(1, -1, 1)
    ph = torch.linspace(0, 2 * math.pi, nv, device=DEV).view(-1, 1, 1)
    shift = 0.3 * torch.sin(ph + 0.37 * (seed % 17))
    s = 20.0 * torch.exp(-2.0 * (u - shift) ** 2 - v ** 2)
    return s.add_(torch.rand(shape, device=DEV, generator=_gen(seed)))


def _residual(shape, seed):
    """Incoming gradient of a projection as a data term gives it, A x - b: smooth structure of both signs
    (what the image still lacks) and measurement noise."""
    s = _soft_sino(shape, seed)
    return s.sub_(0.7 * _soft_sino(shape, seed + 3)).mul_(0.1)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "pair":
        k = _cone(c)
        return dict(kind=kind, geom=ops.ConeBeam(**k), flags=_flags(c),
                    x=_phantom(_vol_shape(k), seed).requires_grad_(),
                    g=_residual(_sino_shape(k), seed))
    if kind == "fdk":
        k = _cone(c)
        geom = ops.ConeBeam(**k)
        return dict(kind=kind, geom=geom, window=c["window"],
                    parker=ops.parker_direction(geom) if c["short"] else 0, sino=_soft_sino(_sino_shape(k), seed))
    if kind == "lor":
        shape = (c["nx"], c["ny"], c["nz"])
        lors = _ring_lines(c, seed)
        return dict(kind=kind, shape=shape, lors=lors, order=ops.lor_order(lors, shape) if c["ordered"] else None,
                    vol=_phantom(shape[::-1], seed),
                    vals=torch.rand(c["lines"], device=DEV, generator=_gen(seed + 1)))
    if kind == "motion":
        geoms = [ops.ConeBeam(**k) for k in _motion_cones(c)]
        return dict(kind=kind, geoms=geoms, x=_phantom((c["n"],) * 3, seed).requires_grad_(),
                    fields=[[f.requires_grad_() for f in m] for m in _fields(c, seed)],
                    g=[_residual(q.sino_shape, seed + 1 + i) for i, q in enumerate(geoms)])
    if kind == "dd":
        geom = ops.DDGeometry((c["nx"], c["ny"], c["nz"]), _angles(c), c["sad"], c["sid"], c["na"], c["px"], c["nb"],
                              c["px"])
        return dict(kind=kind, geom=geom, flags=0 if c["weight"] else _lib.FDK_NO_WEIGHT,
                    x=_phantom(geom.vol_shape, seed).requires_grad_(),
                    g=_residual(geom.proj_shape, seed))
    if kind == "batch":
        geoms = [ops.ConeBeam(**k) for k in _batch_cones(c)]
        vols = [_phantom(q.vol_shape, seed + i, 3) for i, q in enumerate(geoms)]
        grads = [_residual(q.sino_shape, seed + i) for i, q in enumerate(geoms)]
        plan = BatchProjector(geoms, [v.clone() for v in vols], grads=[g.clone() for g in grads])
        return dict(kind=kind, plan=plan, x=[v.requires_grad_() for v in vols], g=grads)
    k = _cone(c)
    geom = ops.ConeBeam(**k)
    b = ops.cb_forward(_phantom(_vol_shape(k), seed), geom, _lib.LINE_INTEGRAL)
    b += 0.01 * torch.randn(b.shape, device=DEV, generator=_gen(seed))
    return dict(kind="solve", solver=c["solver"], geom=geom, b=b, iters=c["iters"])


# ---------------- one pass ----------------

def run(s):
    kind = s["kind"]
    if kind == "pair":
        sino = nb.project(s["x"], s["geom"], s["flags"])
        (grad,) = torch.autograd.grad(sino, s["x"], s["g"])
        return sino, grad
    if kind == "fdk":
        return recon.fdk(s["sino"], s["geom"], s["window"], s["parker"])
    if kind == "lor":
        return (ops.lor_forward(s["lors"], s["vol"], s["shape"], order=s["order"]),
                ops.lor_backward(s["lors"], s["vals"], s["shape"], order=s["order"]))
    if kind == "motion":
        sinos = recon.motion_project(s["x"], s["fields"], s["geoms"])
        leaves = [s["x"]] + [f for m in s["fields"] for f in m]
        return sinos, torch.autograd.grad(sinos, leaves, s["g"])
    if kind == "dd":
        proj = ops.dd_project(s["x"], s["geom"], s["flags"])
        (grad,) = torch.autograd.grad(proj, s["x"], s["g"])
        return proj, grad
    if kind == "batch":
        sinos = batch_project(s["plan"], s["x"])
        return sinos, torch.autograd.grad(sinos, s["x"], s["g"])
    solve = recon.sirt if s["solver"] == "sirt" else recon.cg
    return solve(s["b"], s["geom"], s["iters"])


# ---------------- work of one pass ----------------

def _contributions(k):
    """Ray-voxel contributions of one projection: rays through each voxel times the two voxels a slab is split over."""
    nx, ny, nz = k["shape"]
    vx, vz = k["size"][0] / nx, k["size"][2] / nz
    mag = k["src_det"] / k["src_iso"]
    da = k["da"] * (k["src_det"] if k["det_kind"] == "cyl" else 1.0)
    cover = min(1.0, k["na"] * da / (mag * nx * vx)) * min(1.0, k["nb"] * k["db"] / (mag * nz * vz))
    return nx * ny * nz * len(k["angles"]) * (mag * vx / da) * (mag * vz / k["db"]) * cover


def _pair_work(k):
    data = 4.0 * (2 * math.prod(k["shape"]) + 2 * math.prod(_sino_shape(k)))
    return data, 4.0 * _contributions(k)


def work(case):
    c, kind = case, case["kind"]
    if kind == "pair":
        b, f = _pair_work(_cone(c))
    elif kind == "fdk":
        k = _cone(c)
        length = max(64, 1 << (2 * c["na"] - 1).bit_length())
        vox = math.prod(k["shape"])
        b = 4.0 * (math.prod(_sino_shape(k)) + vox)
        f = 10.0 * vox * c["nv"] + 5.0 * length * math.log2(length) * c["nv"] * c["nb"]
    elif kind == "lor":
        vox = c["nx"] * c["ny"] * c["nz"]
        b = 4.0 * (2 * 8 * c["lines"] + 2 * vox)
        f = 4.0 * c["lines"] * 0.9 * max(c["nx"], c["ny"])
    elif kind == "motion":
        parts = [_pair_work(k) for k in _motion_cones(c)]
        vox = c["n"] ** 3
        b = sum(p[0] for p in parts) + 4.0 * vox * c["phases"] * 6
        f = sum(p[1] for p in parts) + 60.0 * vox * c["phases"]
    elif kind == "dd":
        k = dict(shape=(c["nx"], c["ny"], c["nz"]), size=(c["nx"], c["ny"], c["nz"]), angles=range(c["nv"]),
                 src_iso=c["sad"], src_det=c["sid"], na=c["na"], da=c["px"], nb=c["nb"], db=c["px"], det_kind="flat")
        b, f = _pair_work(k)
        f *= 2
    elif kind == "batch":
        parts = [_pair_work(k) for k in _batch_cones(c)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    else:
        b, f = _pair_work(_cone(c))
        f *= c["iters"] + 1
    return {"bytes": b, "flops": f}


# ---------------- the same in float64, without the package's operators ----------------

F64 = torch.float64
MOST_EXACT = 4e10            # ray-slab pairs of the float64 walk: about ten seconds
CHUNK = 6_000_000            # values per temporary


def _f32(*v):
    """Parameters as the geometry structs carry them (float32)."""
    out = [float(np.float32(x)) for x in v]
    return out if len(out) > 1 else out[0]


def _walk64(shape, size, p1, p2, line=False, tie_gt=False, skip_short=False, q5=False):
    """Slab-split walk of rays p1 -> p2 ([3][N], float64) through a centred grid (nx, ny, nz) of extent
    `size`: yields (rays, voxel index [S, N'], weight [S, N']) with zero weights outside the grid."""
    nx, ny, nz = shape
    sx, sy, sz = (_f32(s) for s in size)
    dx = sx / nx
    dy, dz = sy / ny / dx, sz / nz / dx
    a, b = [v / dx for v in p1], [v / dx for v in p2]
    xd, yd, zd = (b[i] - a[i] for i in range(3))
    xy2 = xd * xd + yd * yd
    L = (xy2 + zd * zd).sqrt()
    xdrive = (xd.abs() > yd.abs()) if tie_gt else (xd.abs() >= yd.abs())
    keep = xy2 >= 100.0 if skip_short else torch.ones_like(xdrive)
    for drive in (True, False):
        rays = torch.nonzero((xdrive == drive) & keep).view(-1)
        if not rays.numel():
            continue
        A, D, l = [v[rays] for v in a], [v[rays] for v in (xd, yd, zd)], L[rays]
        i, j = (0, 1) if drive else (1, 0)
        nu, nv = (nx, ny) if drive else (ny, nx)
        su, sv, sw = (1, nx, nx * ny) if drive else (nx, 1, nx * ny)
        kv, kw = D[j] / D[i], D[2] / D[i]
        dv = dy if drive else 1.0
        W = (1 + kv * kv + kw * kw).sqrt() * dx
        if not line:
            W = W / l / l
        step = max(1, CHUNK // rays.numel())
        for k0 in range(0, nu, step):
            k = torch.arange(k0, min(nu, k0 + step), device=DEV, dtype=F64).view(-1, 1)
            t = k - nu / 2 - A[i]
            qa, qb = (A[j] + kv * t) / dv + nv / 2, (A[j] + kv * (t + 1)) / dv + nv / 2
            q1, q2 = torch.minimum(qa, qb), torch.maximum(qa, qb)
            v1, v2 = q1.floor(), q2.floor()
            vx = v1 != v2
            rv = torch.where(vx, (v2 - q1) / (q2 - q1), 1.0)
            qa, qb = (A[2] + kw * t) / dz + nz / 2, (A[2] + kw * (t + 1)) / dz + nz / 2
            q1, q2 = torch.minimum(qa, qb), torch.maximum(qa, qb)
            w1, w2 = q1.floor(), q2.floor()
            wx = w1 != w2
            rw = torch.where(wx, (w2 - q1) / (q2 - q1), 1.0)
            adm = (v1 < nv) & (w1 < nz) & (v1 >= -vx.double()) & (w1 >= -wx.double())
            first = rv > rw
            mid = W / l if q5 and not drive else W
            for sv_, sw_, r, wt in ((v1, w1, torch.minimum(rv, rw), W),
                                    (torch.where(first, v1, v2), torch.where(first, w2, w1), (rv - rw).abs(),
                                     torch.where(vx & wx, mid, W)),
                                    (v2, w2, 1 - torch.maximum(rv, rw), W)):
                ok = adm & (sv_ >= 0) & (sv_ < nv) & (sw_ >= 0) & (sw_ < nz)
                idx = (k * su + sv_.clamp(0, nv - 1) * sv + sw_.clamp(0, nz - 1) * sw).long()
                yield rays, idx, torch.where(ok, r * wt, 0.0)


def _cone_rays(k, iv):
    si, sd, da, db = _f32(k["src_iso"], k["src_det"], k["da"], k["db"])
    ang = float(k["angles"][iv])
    off = float(k["z_offsets"][iv]) if k["z_offsets"] is not None else 0.0
    cs, sn = math.cos(ang), math.sin(ang)
    a = ((torch.arange(k["na"], device=DEV, dtype=F64) + 0.5) * da - k["na"] * da / 2).repeat(k["nb"])
    b = ((torch.arange(k["nb"], device=DEV, dtype=F64) + 0.5) * db - k["nb"] * db / 2).repeat_interleave(k["na"])
    if k["det_kind"] == "cyl":
        x0, y0 = sd * a.cos() - si, sd * a.sin()
    else:
        x0, y0 = torch.full_like(a, sd - si), a
    p1 = [torch.full_like(a, -si * cs), torch.full_like(a, -si * sn), torch.full_like(a, off)]
    return p1, [x0 * cs - y0 * sn, x0 * sn + y0 * cs, b + off]


def _cone64(k, line, vol=None, sino=None):
    """Forward of vol and / or transpose of sino in float64."""
    fwd = torch.zeros(_sino_shape(k), device=DEV, dtype=F64) if vol is not None else None
    bwd = torch.zeros(math.prod(k["shape"]), device=DEV, dtype=F64) if sino is not None else None
    flat = vol.double().reshape(-1) if vol is not None else None
    for iv in range(len(k["angles"])):
        p1, p2 = _cone_rays(k, iv)
        out = fwd[iv].view(-1) if fwd is not None else None
        y = sino[iv].double().reshape(-1) if sino is not None else None
        for rays, idx, w in _walk64(k["shape"], k["size"], p1, p2, line):
            if out is not None:
                out[rays] += (flat[idx] * w).sum(0)
            if bwd is not None:
                bwd.index_add_(0, idx.view(-1), (w * y[rays]).view(-1))
    return fwd, bwd.view(_vol_shape(k)) if bwd is not None else None


def _fdk64(c, k, sino, parker):
    si, sd, da, db = _f32(k["src_iso"], k["src_det"], k["da"], k["db"])
    na, rows, nv = k["na"], k["nb"], len(k["angles"])
    u = (torch.arange(na, device=DEV, dtype=F64) + 0.5) * da - na * da / 2
    v = (torch.arange(rows, device=DEV, dtype=F64) + 0.5) * db - rows * db / 2
    cosw = sd / (sd * sd + u.view(1, -1) ** 2 + v.view(-1, 1) ** 2).sqrt()
    length = max(64, 1 << (2 * na - 1).bit_length())
    nn = torch.arange(-length // 2, length // 2, device=DEV, dtype=F64)
    h = torch.where(nn % 2 != 0, -1.0 / (math.pi * nn) ** 2, 0.0)
    h[length // 2] = 0.25
    H = 2 * torch.fft.rfft(h).abs()
    w = 2 * math.pi * torch.arange(length // 2 + 1, device=DEV, dtype=F64) / length
    win = {"ram-lak": torch.ones_like(w), "shepp-logan": torch.sin(w / 2) / (w / 2), "cosine": torch.cos(w / 2),
           "hamming": 0.54 + 0.46 * torch.cos(w), "hann": (1 + torch.cos(w)) / 2}[c["window"]]
    H[1:] *= win[1:]
    ang = k["angles"].astype(np.float64)
    dbeta = 2 * math.pi / nv
    pk = torch.ones((nv, na), device=DEV, dtype=F64)
    if parker:
        dang = abs(ang[1] - ang[0]) * 180 / math.pi
        dbeta = 2 * math.pi / (180 / dang)
        g = torch.atan(u / sd) * 180 / math.pi
        fan = float((g[-1] - g[0]).abs()) / 2
        i = torch.arange(1, nv + 1, device=DEV, dtype=F64).view(-1, 1)
        p = ((180 / dang - nv) / 2 + i) * dang + parker * g.view(1, -1)
        up = torch.sin(math.pi / 2 * (fan / 2 + p) / fan).clamp(min=0) ** 2
        down = torch.cos(math.pi / 2 * (fan / 2 + p - 180) / fan).clamp(min=0) ** 2
        pk = torch.where((p <= fan / 2) & (p > -fan / 2), pk * up, pk)
        pk = torch.where((p >= 180 - fan / 2) & (p < 180 + fan / 2), pk * down, pk)
        pk = torch.where((p < -fan / 2) | (p > 180 + fan / 2), 0.0, pk)
    scale = 0.5 / da * dbeta / 2 * (sd / si)
    nx, ny, nz = k["shape"]
    sx, sy, sz = (_f32(s) for s in k["size"])
    x = ((torch.arange(nx, device=DEV, dtype=F64) + 0.5) * sx / nx - sx / 2).view(1, -1)
    y = ((torch.arange(ny, device=DEV, dtype=F64) + 0.5) * sy / ny - sy / 2).view(-1, 1)
    z = ((torch.arange(nz, device=DEV, dtype=F64) + 0.5) * sz / nz - sz / 2).view(-1, 1, 1)
    vol = torch.zeros((nz, ny, nx), device=DEV, dtype=F64)
    for iv in range(nv):
        row = sino[iv].double() * cosw * pk[iv]
        f = torch.fft.irfft(torch.fft.rfft(row, length) * H, length)[:, :na] * scale
        f = f.reshape(-1)
        cs, sn = math.cos(ang[iv]), math.sin(ang[iv])
        xr, yr = x * cs + y * sn, -x * sn + y * cs
        m = sd / (xr + si)
        wt = (si / (si + xr)) ** 2
        a = m * yr / da + na // 2 - 0.5
        b = m * z / db + rows // 2 - 0.5
        ia, ib = a.floor(), b.floor()
        ok = (ia >= 0) & (ia + 1 < na) & (ib >= 0) & (ib + 1 < rows)
        fa, fb = a - ia, b - ib
        i0 = (ib.clamp(0, rows - 2) * na + ia.clamp(0, na - 2)).long()
        val = (f[i0] * (1 - fa) + f[i0 + 1] * fa) * (1 - fb) + (f[i0 + na] * (1 - fa) + f[i0 + na + 1] * fa) * fb
        vol += torch.where(ok, val * wt, 0.0)
    return vol


def _lor64(c, s):
    p = [s["lors"][i].double() for i in range(6)]
    flat, vals = s["vol"].double().reshape(-1), s["vals"].double()
    fwd = torch.zeros(c["lines"], device=DEV, dtype=F64)
    bwd = torch.zeros(flat.numel(), device=DEV, dtype=F64)
    shape, size = s["shape"], s["shape"]
    part = 200_000
    for i in range(0, c["lines"], part):
        p1, p2 = [v[i:i + part] for v in p[:3]], [v[i:i + part] for v in p[3:]]
        for rays, idx, w in _walk64(shape, size, p1, p2, tie_gt=True, skip_short=True, q5=True):
            fwd[i + rays] += (flat[idx] * w).sum(0)
        for rays, idx, w in _walk64(shape, size, p1, p2, line=True, tie_gt=True, skip_short=True):
            bwd.index_add_(0, idx.view(-1), (w * vals[i + rays]).view(-1))
    return fwd, bwd.view(s["vol"].shape)


def _taps64(shape, m):
    """Corner indices, fractions and validity of the trilinear samples i + m[i]."""
    nz, ny, nx = shape
    ar = [torch.arange(n, device=DEV, dtype=F64) for n in (nx, ny, nz)]
    pos = [ar[0].view(1, 1, -1) + m[0].double(), ar[1].view(1, -1, 1) + m[1].double(),
           ar[2].view(-1, 1, 1) + m[2].double()]
    low = [p.floor() for p in pos]
    ok = torch.ones(shape, device=DEV, dtype=torch.bool)
    for q, n in zip(low, (nx, ny, nz)):
        ok &= (q > 0) & (q + 1 < n)
    base = torch.where(ok, low[0] + low[1] * nx + low[2] * nx * ny, 0.0).long()
    return base, [p - q for p, q in zip(pos, low)], ok, (1, nx, nx * ny)


def _motion64(c, s):
    x = s["x"].detach().double()
    shape, flat = x.shape, x.reshape(-1)
    gx = torch.zeros_like(flat)
    sinos, gf = [], []
    for k, m, g in zip(_motion_cones(c), s["fields"], s["g"]):
        base, f, ok, st = _taps64(shape, [q.detach() for q in m])
        corners = [(i, j, l) for i in (0, 1) for j in (0, 1) for l in (0, 1)]
        val = {q: flat[torch.where(ok, base + q[0] * st[0] + q[1] * st[1] + q[2] * st[2], 0)] for q in corners}
        wt = [[1 - t, t] for t in f]
        warped = torch.where(ok, sum(val[q] * wt[0][q[0]] * wt[1][q[1]] * wt[2][q[2]] for q in corners), 0.0)
        sino, back = _cone64(k, False, warped, g)
        sinos.append(sino)
        gb = torch.where(ok, back, 0.0)
        for q in corners:
            gx.index_add_(0, torch.where(ok, base + q[0] * st[0] + q[1] * st[1] + q[2] * st[2], 0).view(-1),
                          (gb * wt[0][q[0]] * wt[1][q[1]] * wt[2][q[2]]).view(-1))
        for d in range(3):
            o = [i for i in range(3) if i != d]
            gf.append(gb * sum((2 * q[d] - 1) * val[q] * wt[o[0]][q[o[0]]] * wt[o[1]][q[o[1]]] for q in corners))
    return sinos, [gx.view(shape)] + gf


def _dd64(c, s):
    g = s["geom"]
    nx, ny, nz = g.shape
    sad, sid, d = _f32(c["sad"], c["sid"], c["px"])
    na, rows = c["na"], c["nb"]
    flat, cot = s["x"].detach().double().reshape(-1), s["g"].double()
    fwd = torch.zeros(g.proj_shape, device=DEV, dtype=F64)
    bwd = torch.zeros(flat.numel(), device=DEV, dtype=F64)
    edge = torch.arange(na + 1, device=DEV, dtype=F64) * d - na * d / 2
    mid = (torch.arange(na, device=DEV, dtype=F64) + 0.5) * d - na * d / 2
    zmid = (torch.arange(rows, device=DEV, dtype=F64) + 0.5) * d - rows * d / 2
    for iv, ang in enumerate(g.angles.astype(np.float64)):
        cs, sn = math.cos(ang), math.sin(ang)
        x1, y1 = -sad * cs, -sad * sn
        x21, y21 = (sid - sad) * cs - mid * sn - x1, (sid - sad) * sn + mid * cs - y1
        ex, ey = (sid - sad) * cs - edge * sn - x1, (sid - sad) * sn + edge * cs - y1
        for xd in (True, False):
            cols = torch.nonzero((x21.abs() > y21.abs()) == xd).view(-1)
            if not cols.numel():
                continue
            nu, nt = (nx, ny) if xd else (ny, nx)
            u1, v1 = (x1, y1) if xd else (y1, x1)
            e = (ex, ey) if xd else (ey, ex)
            u21 = (x21 if xd else y21)[cols]
            ul, vl, ur, vr = e[0][cols], e[1][cols], e[0][cols + 1], e[1][cols + 1]
            slopes = [vl / ul, vl / ur, vr / ul, vr / ur]
            length = (x21[cols] ** 2 + y21[cols] ** 2 + zmid.view(-1, 1) ** 2).sqrt() / u21.abs()
            zl, zr = (zmid.view(-1, 1) - d / 2) / u21, (zmid.view(-1, 1) + d / 2) / u21
            y = cot[iv][:, cols]
            acc = torch.zeros((rows, cols.numel()), device=DEV, dtype=F64)
            step = max(1, CHUNK // (rows * cols.numel()))
            for k0 in range(0, nu, step):
                iu = torch.arange(k0, min(nu, k0 + step), device=DEV, dtype=F64).view(-1, 1, 1)
                uc = iu + 0.5 - nu / 2 - u1
                q = [r * uc + v1 + nt // 2 for r in slopes]
                lo = torch.minimum(torch.minimum(q[0], q[1]), torch.minimum(q[2], q[3]))
                hi = torch.maximum(torch.maximum(q[0], q[1]), torch.maximum(q[2], q[3]))
                za, zb = zl * uc + nz // 2, zr * uc + nz // 2
                z1, z2 = torch.minimum(za, zb), torch.maximum(za, zb)
                f1, g1 = lo.floor(), z1.floor()
                spans = int((hi.floor() - f1).max()) + 1, int((z2.floor() - g1).max()) + 1
                for i in range(spans[0]):
                    iv2 = f1 + i
                    wv = (torch.minimum(iv2 + 1, hi) - torch.maximum(iv2, lo)).clamp(min=0) / (hi - lo)
                    wv = torch.where((iv2 >= 0) & (iv2 < nt), wv, 0.0)
                    ix, iy = (iu, iv2) if xd else (iv2, iu)
                    if c["weight"]:
                        den = sad + (ix + 0.5 - nx // 2) * cs + (iy + 0.5 - ny // 2) * sn
                        wv = wv * (sad / den) ** 2
                    col = ix + iy.clamp(0, ny - 1) * nx if xd else ix.clamp(0, nx - 1) + iy * nx
                    for j in range(spans[1]):
                        iz = g1 + j
                        wz = (torch.minimum(iz + 1, z2) - torch.maximum(iz, z1)).clamp(min=0) / (z2 - z1)
                        wt = torch.where((iz >= 0) & (iz < nz), wz * wv * length, 0.0)
                        idx = (col + iz.clamp(0, nz - 1) * (nx * ny)).long()
                        acc += (flat[idx] * wt).sum(0)
                        bwd.index_add_(0, idx.view(-1), (wt * y).view(-1))
            fwd[iv][:, cols] = acc
    return fwd, bwd.view(g.vol_shape)


def _solve64(c, k, b):
    b = b.double()

    def fwd(v):
        return _cone64(k, True, vol=v)[0]

    def bwd(v):
        return _cone64(k, True, sino=v)[1]

    x = torch.zeros(_vol_shape(k), device=DEV, dtype=F64)
    if c["solver"] == "sirt":
        rs, cs = fwd(torch.ones_like(x)), bwd(torch.ones_like(b))
        R, C = torch.where(rs > 0, 1 / rs, 0.0), torch.where(cs > 0, 1 / cs, 0.0)
        for _ in range(c["iters"]):
            x = x + C * bwd(R * (b - fwd(x)))
        return x
    r = bwd(b)
    p, old = r.clone(), (r * r).sum()
    for _ in range(c["iters"]):
        ap = bwd(fwd(p))
        alpha = old / (p * ap).sum()
        x, r = x + alpha * p, r - alpha * ap
        new = (r * r).sum()
        p, old = r + (new / old) * p, new
    return x


def exact(case, seed):
    c, kind = case, case["kind"]

    def slabs(k):
        return math.prod(_sino_shape(k)) * max(k["shape"][:2])

    if kind == "pair":
        k = _cone(c)
        if slabs(k) > MOST_EXACT:
            return None
        s = prepare(case, seed)
        return _cone64(k, c["line"], s["x"].detach(), s["g"])
    if kind == "fdk":
        s = prepare(case, seed)
        return _fdk64(c, _cone(c), s["sino"], s["parker"])
    if kind == "lor":
        return _lor64(c, prepare(case, seed))
    if kind == "motion":
        return _motion64(c, prepare(case, seed))
    if kind == "dd":
        return _dd64(c, prepare(case, seed))
    if kind == "batch":
        s = prepare(case, seed)
        both = [_cone64(k, False, x.detach(), g) for k, x, g in zip(_batch_cones(c), s["x"], s["g"])]
        return [f for f, _ in both], [g for _, g in both]
    k = _cone(c)
    if slabs(k) * (c["iters"] + 1) > MOST_EXACT:
        return None
    return _solve64(c, k, prepare(case, seed)["b"])
