"""The work that a user of this framework has it do, as cases that can be timed.

Every case runs one of the seeded systems of the package's geometry module through a public
entry point of its Python binding.  The seed moves the image by a fraction of a millimetre and
varies the attenuation coefficients by a few percent, as calibrated systems differ from their
drawings.

  listed()             the named cases; each states below what it stands for
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what a program holds before the call: contexts, plans, inputs, outputs
  run(state)           one pass
  work(case)           bytes and operations that the pass cannot do without
  exact(case, seed)    the pass's results in 64 bits, from plain torch
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "gpu-based-system-matrix-calculation-for-spect-pet_b200")


def _load(name, path):
    if name in sys.modules:
        return sys.modules[name]
    spec = importlib.util.spec_from_file_location(name, path)
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    spec.loader.exec_module(mod)
    return mod


geometry = _load("sysmat_geometry", os.path.join(PKG, "geometry.py"))
sysmat = _load("sysmat_binding", os.path.join(PKG, "sysmat.py"))

MODES = {"reference": sysmat.MODE_REFERENCE, "precise": sysmat.MODE_PRECISE, "fp64": sysmat.MODE_FP64,
         "local": sysmat.MODE_LOCAL}


# ---------------------------------------------------------------------------------------
# The cases.  path: the entry point; system: the geometry; det, dets / vox, voxs: the block of
# detector rows and of voxels.

def listed():
    return [
        # the smallest matrix: a bench-top prototype (36 crystals, 128 voxels), as unit tests and
        # quick design checks compute it; launches and latency count
        dict(name="pe_prototype", path="pe", mode="reference", system="mini", layers=1, rotated=True, rot=0,
             det=0, dets=36, vox=0, voxs=128),
        # the reference-compatible host call (arrays in, matrix out) on the plain PE system, a new
        # system each call
        dict(name="pe_host_call", path="host", system="config1"),
        # one crystal block of a production plane: the headline workload
        dict(name="pe_production_plane", path="pe", mode="reference", system="config2", rot=0, det=1984, dets=128,
             vox=16 * 9216, voxs=9216),
        # the voxel columns that one of many ranks owns: a ragged strip of voxels, all crystals
        dict(name="pe_rank_columns", path="pe", mode="reference", system="config3", rot=0, det=0, dets=1024,
             vox=19147, voxs=301),
        # accurate modes on a ragged block of the production system
        dict(name="pe_fp64_block", path="pe", mode="fp64", system="config2", rot=0, det=77, dets=61, vox=148001,
             voxs=2303),
        dict(name="pe_local_block", path="pe", mode="local", system="config2", rot=0, det=2048, dets=64,
             vox=15 * 9216, voxs=2304),
        # the production system with its stated sampling (2x8x2 sub-elements, 2x2x2 sources)
        dict(name="pe_sampled", path="sampled", mode="precise", system="config2", rot=0, det=2000, dets=96,
             vox=16 * 9216, voxs=4608, div="2,8,2", sub="2,2,2"),
        # a design sweep: 16 collimators, each at one of its rotations, 8 crystal rows of 8 planes
        dict(name="pe_design_sweep", path="batch", mode="reference", system="config4", designs=16, det=500, dets=8,
             vox=4096, voxs=8192),
        # scatter of a new system: relationship bitmaps, pair tables, then a block of voxels
        dict(name="scatter_new_system", path="scatter", system="config3", parts=3, det=0, dets=1024, vox=18433,
             voxs=768),
        # forward and back projection of one crystal block (an MLEM subset)
        dict(name="projector_pair", path="projector", system="config5", det=1152, dets=24),
        # the gradient of the projection with respect to the collimator (calibration)
        dict(name="projector_gradient", path="gradient", system="config5", det=1100, dets=96),
        # scatter points on a grid inside crystals and septa
        dict(name="scatter_grid", path="grid", system="config3", parts=3, cell=0.5, det=512, dets=64, vox=18500,
             voxs=24),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


SIZES = {"mini": (36, 128), "config1": (256, 1024), "config2": (4096, 294912), "config3": (1024, 36864),
         "config4": (1024, 16384), "config5": (2304, 65536)}
# matrix elements that a drawn block holds at most, by path and mode
MOST = {"reference": 1000000, "precise": 1000000, "fp64": 130000, "local": 130000, "sampled": 400000}


def _block(rng, system, most):
    """A block of detector rows x voxels of `system` with at most `most` elements."""
    n_det, n_vox = SIZES[system]
    dets = _log_int(rng, 1, min(n_det, most // 64))
    voxs = _log_int(rng, 1, min(n_vox, most // dets))
    return dict(det=rng.randrange(n_det - dets + 1), dets=dets, vox=rng.randrange(n_vox - voxs + 1), voxs=voxs)


def draw(rng):
    path = rng.choice(["pe", "pe", "pe", "pe", "host", "sampled", "batch", "scatter", "projector", "gradient", "grid"])
    if path == "pe":
        mode = rng.choice(["reference", "reference", "reference", "precise", "fp64", "local"])
        system = rng.choice(["mini", "config1", "config2", "config3", "config4"])
        case = dict(path="pe", mode=mode, system=system, rot=rng.randrange(12) if system == "config4" else 0)
        if system == "mini":
            case.update(layers=rng.randint(1, 3), rotated=rng.random() < 0.5)
        case.update(_block(rng, system, MOST[mode]))
        return case
    if path == "host":
        return dict(path="host", system="mini", layers=rng.randint(1, 3), rotated=rng.random() < 0.5,
                    side=rng.randint(4, 24))
    if path == "sampled":
        mode = rng.choice(["precise", "local"])
        case = dict(path="sampled", mode=mode, system=rng.choice(["config1", "config2"]), rot=0,
                    div=rng.choice(["4,4,4", "2,8,2", "3,5,2"]), sub=rng.choice(["1,1,1", "2,2,2", "1,3,2"]))
        case.update(_block(rng, case["system"], MOST["sampled"] // (1 if mode == "precise" else 2)))
        return case
    if path == "batch":
        return dict(path="batch", mode=rng.choice(["reference", "precise"]), system="config4",
                    designs=rng.randint(2, 16), det=rng.randrange(1000), dets=_log_int(rng, 1, 24),
                    vox=rng.randrange(8192), voxs=_log_int(rng, 64, 4096))
    if path == "scatter":
        return dict(path="scatter", system="config3", parts=rng.randint(1, 3), det=rng.randrange(500),
                    dets=_log_int(rng, 16, 512), vox=rng.randrange(30000), voxs=_log_int(rng, 16, 2304))
    if path == "projector":
        return dict(path="projector", system="config5", det=rng.randrange(2270), dets=_log_int(rng, 2, 24))
    if path == "gradient":
        return dict(path="gradient", system="config5", det=rng.randrange(2100), dets=_log_int(rng, 8, 128))
    return dict(path="grid", system="config3", parts=rng.randint(1, 3), cell=rng.choice([0.5, 0.7]),
                det=rng.randrange(900), dets=_log_int(rng, 8, 100), vox=rng.randrange(30000),
                voxs=_log_int(rng, 2, 40))


# ---------------------------------------------------------------------------------------
# Systems and inputs.

def _varied(geo, seed, salt=0):
    """`geo` with the image moved by up to 0.3 mm and the coefficients varied by up to 2 %."""
    rng = np.random.default_rng([seed & 0x7FFFFFFF, salt])
    img, col, det = geo.image.copy(), geo.collimator.copy(), geo.detector.copy()
    img[8:11] += rng.uniform(-0.3, 0.3, 3).astype(np.float32)
    w = np.float32(1 + rng.uniform(-0.02, 0.02))
    c = np.float32(1 + rng.uniform(-0.02, 0.02))
    for m in range(geo.n_layers):
        col[10 * (m + 1) + 5:10 * (m + 1) + 8] *= w
    det[1:1 + 12 * geo.n_det].reshape(-1, 12)[:, 6:9] *= c
    return geometry.Geometry(geo.name, col, det, img, geo.physics, dict(geo.meta))


def _system(case, seed):
    kind = case["system"]
    if kind == "mini":
        side = case.get("side", 6)
        geo = geometry.mini(seed=3, rotated=bool(case.get("rotated")), layers=int(case.get("layers", 1)),
                            nvox=(8, 8, 2), ncry=(side, side), nholes=max(5, side))
    elif kind == "config5":
        geo = geometry.config5()[0]
    elif kind == "config4":
        geo = geometry.config4(8)[5]
    else:
        geo = {"config1": geometry.config1, "config2": geometry.config2, "config3": geometry.config3}[kind]()
    return _varied(geo, seed)


def _ints(text):
    return tuple(int(x) for x in text.split(","))


def _plain_pe(geo, seed, v0, nv):
    """A photoelectric matrix of the system's size, n_det x n_vox float32 on the GPU, zero but for
    the voxel columns that are read: solid angle of the crystal's face times the absorbed
    share, through a collimator that passes axial rays, with a seeded spread."""
    D, V = geo.n_det, geo.n_vox
    d = torch.from_numpy(geo.detector[1:1 + 12 * D].reshape(D, 12).astype(np.float64)).cuda()
    I = _voxels(geo, 0.0, v0, nv)
    fov = float(geo.image[11])
    dx, dz = d[:, None, 0] - I[None, :, 0], d[:, None, 2] - I[None, :, 2]
    dy = d[:, None, 1] + fov - I[None, :, 1]
    r2 = dx * dx + dy * dy + dz * dz
    tan2 = (dx * dx + dz * dz) / (dy * dy)
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)
    spread = torch.rand((D, nv), generator=g, device="cuda", dtype=torch.float64)
    val = d[:, None, 3] * d[:, None, 5] / (4 * math.pi * r2) * 0.6 * torch.exp(-20 * tan2.clamp(max=0.7) - 2 * spread)
    pe = torch.zeros((D, V), dtype=torch.float32, device="cuda")
    pe[:, v0:v0 + nv] = val.float()
    return pe


def _activity(case, seed):
    x = geometry.ellipsoid_phantom((64, 64, 16), (1.0, 1.0, 1.0), 5, 5)
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 1])
    x = x * rng.uniform(0.8, 1.2, x.size).astype(np.float32)
    u = rng.uniform(0.5, 1.5, case["dets"]).astype(np.float32)
    return torch.from_numpy(x).cuda(), torch.from_numpy(u).cuda()


class State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    path = case["path"]
    if path == "host":
        geo = _system(case, seed)
        return State(case=case, geo=geo, dst=np.zeros((geo.n_det, geo.n_vox), dtype=np.float32))
    if path == "batch":
        designs = geometry.config4(case["designs"])
        geos = [_varied(g, seed, k + 1) for k, g in enumerate(designs)]
        ctxs = [sysmat.Context(g) for g in geos]
        outs = [torch.zeros((case["dets"], case["voxs"]), dtype=torch.float32, device="cuda") for _ in ctxs]
        items = [(k, float((7 * k) % geos[k].n_rot), case["det"], case["dets"], case["vox"], case["voxs"], outs[k])
                 for k in range(len(ctxs))]
        return State(case=case, ctxs=ctxs, outs=outs, plan=sysmat.BatchPlan(ctxs, items))
    geo = _system(case, seed)
    ctx = sysmat.Context(geo)
    s = State(case=case, ctx=ctx)
    if path in ("projector", "gradient"):
        s.x, s.u = _activity(case, seed)
        return s
    s.out = torch.zeros((case["dets"], case["voxs"]), dtype=torch.float32, device="cuda")
    if path == "scatter":
        s.pe = _plain_pe(geo, seed, case["vox"], case["voxs"])
    return s


def run(s):
    c, path = s.case, s.case["path"]
    if path == "host":
        sysmat.PESysMatGen(s.geo.collimator, s.geo.detector, s.geo.image, s.dst)
        return s.dst
    if path == "batch":
        s.plan.run(MODES[c["mode"]])
        return s.outs
    if path == "projector":
        p = s.ctx.project(s.x, det_begin=c["det"], det_count=c["dets"])
        q = s.ctx.backproject(s.u, det_begin=c["det"], det_count=c["dets"])
        return {"p": p, "q": q}
    if path == "gradient":
        return s.ctx.vjp(s.x, s.u, det_begin=c["det"], det_count=c["dets"])
    block = dict(det_begin=c["det"], det_count=c["dets"], vox_begin=c["vox"], vox_count=c["voxs"])
    if path == "pe":
        return s.ctx.pe(s.out, rotation=c["rot"], mode=MODES[c["mode"]], **block)
    if path == "sampled":
        return s.ctx.pe_sampled(s.out, _ints(c["div"]), _ints(c["sub"]), rotation=c["rot"], mode=MODES[c["mode"]],
                                **block)
    if path == "scatter":
        crystal = s.ctx.bitmap_crystal() if c["parts"] & 1 else None
        collimator = s.ctx.bitmap_collimator() if c["parts"] & 2 else None
        s.ctx.scatter_prepare(crystal, collimator, parts=c["parts"])
        s.ctx.scatter(s.out, s.pe if c["parts"] & 1 else None, parts=c["parts"], **block)
        return {"crystal": crystal, "collimator": collimator, "scatter": s.out}
    return s.ctx.scatter_grid(s.out, parts=c["parts"], cell=c["cell"], **block)


# ---------------------------------------------------------------------------------------
# What a pass cannot do without.  Operations per ray of the photoelectric element (the
# reference's formulas: 104 for the sub-element, 25 per box chord, 61 per crossed hole, 45 per
# crossed crystal, with rough mean crossings of each system), per scatter item (about 250), and
# per grid item (about 250); bytes: the parameters and inputs read once, the results written once.

CROSSED = {"mini": (1, 1), "config1": (2, 1), "config2": (5, 2), "config3": (4, 2), "config4": (4, 2),
           "config5": (3, 2)}


def _ray_flops(system, layers):
    h, c = CROSSED[system]
    return 104 + 25 * (layers + 3) + 61 * h + 45 * c


def work(case):
    path, system = case["path"], case["system"]
    params = 4 * (80000 + 80000 + 200)
    ray = _ray_flops(system, case.get("layers", 1))
    if path == "host":
        n = 262144 if system == "config1" else case["side"] ** 2 * 128
        return {"bytes": params + 4 * n, "flops": 1024 * n * ray}
    if path == "projector":
        active = int(np.count_nonzero(geometry.ellipsoid_phantom((64, 64, 16), (1.0, 1.0, 1.0), 5, 5)))
        return {"bytes": params + 12 * 65536 + 12 * case["dets"], "flops": 1024 * case["dets"] * (65536 + active) * ray}
    if path == "gradient":
        active = int(np.count_nonzero(geometry.ellipsoid_phantom((64, 64, 16), (1.0, 1.0, 1.0), 5, 5)))
        return {"bytes": params + 4 * 65536 + 4 * case["dets"], "flops": 1024 * case["dets"] * active * 1.5 * ray}
    n = case["dets"] * case["voxs"]
    if path == "batch":
        n *= case["designs"]
        return {"bytes": case["designs"] * params + 4 * n, "flops": 1024 * n * ray}
    if path == "pe":
        return {"bytes": params + 4 * n, "flops": 1024 * n * ray}
    if path == "sampled":
        rays = math.prod(_ints(case["div"])) * math.prod(_ints(case["sub"]))
        return {"bytes": params + 4 * n, "flops": rays * n * ray}
    if path == "scatter":
        points = 1024 * ((case["parts"] & 1) + (case["parts"] >> 1))
        words = (524800 * 1024 // 32) * (case["parts"] & 1) + (1 << 25) * (case["parts"] >> 1)
        return {"bytes": params + 4 * words + 4 * n + 4 * 1024 * case["voxs"], "flops": 250 * n * points}
    cell = case["cell"]
    cells = [math.ceil(s / cell - 1e-9) for s in (2.0, 6.0, 2.0)]
    septa = [math.ceil(s / cell - 1e-9) for s in (64.0, 10.0, 64.0)]
    points = 1024 * math.prod(cells) * (case["parts"] & 1) + 0.8 * math.prod(septa) * (case["parts"] >> 1)
    return {"bytes": params + 4 * n, "flops": 250 * n * points}


# ---------------------------------------------------------------------------------------
# The results in 64 bits: the photoelectric element and the scatter item of the reference's
# formulas in double, over all rays of all (element, object) pairs that pass its cone test.

EPS = float(np.float32(0.001))


def _voxels(geo, rotation, v0, nv, frac=(0.5, 0.5, 0.5)):
    """Source points of voxels v0 .. v0+nv-1 at fractions `frac` of the voxel, (nv, 3) double."""
    im = [float(x) for x in geo.image]
    nx, ny, nz = int(im[0]), int(im[1]), int(im[2])
    v = torch.arange(v0, v0 + nv, device="cuda", dtype=torch.int64)
    x = ((v % nx).double() - nx / 2 + frac[0]) * im[3] + im[8]
    y = ((v // nx % ny).double() - ny / 2 + frac[1]) * im[4] + im[9]
    z = ((v // (nx * ny)).double() - nz / 2 + frac[2]) * im[5] + im[10]
    a = rotation * im[7]
    return torch.stack([x * math.cos(a) - y * math.sin(a), x * math.sin(a) + y * math.cos(a), z], dim=1)


def _tables(geo):
    D, H = geo.n_det, geo.n_holes
    det = torch.from_numpy(geo.detector[1:1 + 12 * D].reshape(D, 12).astype(np.float64)).cuda()
    det[:, 1] += float(geo.image[11])
    hole = torch.from_numpy(geo.collimator[100:100 + 9 * H].reshape(H, 9).astype(np.float64)).cuda()
    hole[:, 1:3] += float(geo.image[11])
    layers, h = [], 0
    for m in range(geo.n_layers):
        n, w, t, ht, yo, mu = (float(x) for x in geo.collimator[10 * (m + 1):10 * (m + 1) + 6])
        y = float(geo.image[11]) + yo
        layers.append(((-w / 2, y - t / 2, -ht / 2), (w / 2, y + t / 2, ht / 2), t, mu, h, h + int(n)))
        h += int(n)
    return det, hole, layers


def _slabs(p, q, lo, hi):
    """Entry and exit parameters (lengths from p) of segment p -> q in the box, and its length;
    p, q: three broadcastable components each."""
    dl = [b - a for a, b in zip(p, q)]
    tio = (dl[0] ** 2 + dl[1] ** 2 + dl[2] ** 2).sqrt()
    tmin = tmax = None
    for a in range(3):
        inv = tio / dl[a]
        u, w = (lo[a] - p[a]) * inv, (hi[a] - p[a]) * inv
        e, x = torch.minimum(u, w), torch.maximum(u, w)
        tmin = e if tmin is None else torch.maximum(tmin, e)
        tmax = x if tmax is None else torch.minimum(tmax, x)
    return tmin, tmax, tio


def _crossing(p, q, lo, hi):
    """Chord of a full crossing of the box strictly between the segment's ends, else 0."""
    a, b, tio = _slabs(p, q, lo, hi)
    ok = (b - a >= EPS) & (a < tio) & (b < tio) & (a > EPS) & (b > EPS)
    return torch.where(ok, b - a, torch.zeros_like(a))


def _to_end(p, q, lo, hi):
    """Chord from the box entry to the segment's end inside the box."""
    a, b, tio = _slabs(p, q, lo, hi)
    length = torch.minimum(b, tio) - torch.where(a > EPS, a, torch.zeros_like(a))
    ok = (b - a >= EPS) & (a < tio) & (b > EPS)
    return torch.where(ok, length, torch.zeros_like(a))


def _cylinder(p, q, xc, y1, y2, zc, r):
    dl = [b - a for a, b in zip(p, q)]
    tio = (dl[0] ** 2 + dl[1] ** 2 + dl[2] ** 2).sqrt()
    kx, ky, kz = dl[0] / tio, dl[1] / tio, dl[2] / tio
    ta, tb = (y1 - p[1]) / ky, (y2 - p[1]) / ky
    ox, oz = p[0] - xc, p[2] - zc
    fl = (ox + kx * ta) ** 2 + (oz + kz * ta) ** 2 <= r * r
    fr = (ox + kx * tb) ** 2 + (oz + kz * tb) ** 2 <= r * r
    kk = kx * kx + kz * kz
    disc = kk * r * r - (kx * oz - kz * ox) ** 2
    b, root = -(kx * ox + kz * oz), disc.clamp(min=0).sqrt()
    t1, t2 = (b - root) / kk, (b + root) / kk
    ea, eb = torch.where(fl, ta, t1), torch.where(fr, tb, t2)
    ok = (fl & fr) | ((disc > 1e-5) & (fl | fr | ((t1 >= ta) & (t2 <= tb))))
    ok &= (ea > 1e-4) & (eb > 1e-4) & (ea < tio) & (eb < tio)
    return torch.where(ok, eb - ea, torch.zeros_like(ea))


def _pe_exact(geo, rotation, d0, nd, v0, nv, div=(8, 16, 8), sub=(1, 1, 1), voxels=None):
    """Photoelectric elements [d0, d0+nd) x [v0, v0+nv) (or the voxel list) in double."""
    total = None
    for p in range(math.prod(sub)):
        j = (p % sub[0], p // sub[0] % sub[1], p // (sub[0] * sub[1]))
        frac = tuple((j[a] + 0.5) / sub[a] for a in range(3))
        if voxels is None:
            I = _voxels(geo, rotation, v0, nv, frac)
        else:
            I = _voxels(geo, rotation, 0, geo.n_vox, frac)[voxels]
        part = _pe_from(geo, I, d0, nd, div)
        total = part if total is None else total + part
    return total / math.prod(sub)


def _pe_from(geo, I, d0, nd, div):
    det, hole, layers = _tables(geo)
    nv, n_sub = I.shape[0], math.prod(div)
    out = torch.zeros((nd, nv), dtype=torch.float64, device="cuda")
    s = torch.arange(n_sub, device="cuda")
    fx = ((s // div[1] % div[0]).double() + 0.5) / div[0]
    fy = ((s % div[1]).double() + 0.5) / div[1]
    fz = ((s // (div[0] * div[1])).double() + 0.5) / div[2]
    diag = 0.5 * det[:, 3:6].square().sum(1).sqrt()
    h_mid, h_rad = 0.5 * (hole[:, 1] + hole[:, 2]), 0.5 * (4 * hole[:, 4] ** 2 + (hole[:, 1] - hole[:, 2]) ** 2).sqrt()
    centre = torch.cat([torch.stack([hole[:, 0], h_mid, hole[:, 3]], 1), det[:, :3]])
    radius = torch.cat([h_rad, diag])
    foot = torch.cat([hole[:, 4], 0.5 * (det[:, 3] ** 2 + det[:, 5] ** 2).sqrt()])
    near = torch.cat([hole[:, 1], det[:, 1] - 0.5 * det[:, 4]])
    far = torch.cat([hole[:, 2], det[:, 1] + 0.5 * det[:, 4]])
    H = hole.shape[0]
    step = max(1, min(nv, int(4e9 / (centre.shape[0] * 8 * 8))))
    for d in range(d0, d0 + nd):
        P, (w, t, h), mu_t, mu_pe, rot = det[d, :3], [float(x) for x in det[d, 3:6]], float(det[d, 6]), \
            float(det[d, 7]), float(det[d, 10])
        if mu_t <= 0.01:
            continue
        c, sn = math.cos(rot), math.sin(rot)
        xs, ys, zs = (fx - 0.5) * w, (fy - 0.5) * t, (fz - 0.5) * h
        X, Y, Z = P[0] + (xs * c - zs * sn), P[1] + ys, P[2] + (xs * sn + zs * c)
        for b in range(0, nv, step):
            E = I[b:b + step]
            L = (P - E).norm(dim=1)
            u = (P - E) / L[:, None]
            off = centre[None] - E[:, None]
            Lo = off.norm(dim=2)
            keep = (off / Lo[..., None] - u[:, None]).norm(dim=2) <= radius[None] / Lo + (diag[d] / L)[:, None]
            keep[:, H + d] = False
            # objects whose slopes cannot meet the crystal's rays have zero chords
            dy = Y[None] - E[:, 1:2]
            for a, R in ((0, X), (2, Z)):
                sl = (R[None] - E[:, a:a + 1]) / dy
                lo, hi = sl.min(1).values[:, None] - 1e-4, sl.max(1).values[:, None] + 1e-4
                yn, yf = near[None] - E[:, 1:2], far[None] - E[:, 1:2]
                a0, a1 = off[..., a] - foot[None], off[..., a] + foot[None]
                o_lo = torch.minimum(a0 / yn, a0 / yf)
                o_hi = torch.maximum(a1 / yn, a1 / yf)
                keep &= ((o_lo <= hi) & (o_hi >= lo)) | (yn < 1.0)
            e_idx, o_idx = keep.nonzero(as_tuple=True)
            counts = torch.bincount(e_idx, minlength=E.shape[0]).cumsum(0).tolist()
            start, k0 = 0, 0
            while start < E.shape[0]:          # voxels whose (pair, ray) work fits
                stop = start + 1
                while stop < E.shape[0] and (counts[stop] - k0) * n_sub <= 4e7 and (stop - start) * n_sub <= 2e7:
                    stop += 1
                k1 = counts[stop - 1]
                out[d - d0, b + start:b + stop] = _pe_rays(
                    E[start:stop], e_idx[k0:k1] - start, o_idx[k0:k1], H, det, hole, layers, (X, Y, Z), (xs, ys, zs),
                    (fx, fy, fz), div, d)
                start, k0 = stop, k1
    return out


def _pe_rays(E, e, o, H, det, hole, layers, Q, qs, frac, div, d):
    """Sum over the rays E[i] -> Q of one crystal's contributions; (e, o): the kept objects."""
    w, t, h, mu_t, mu_pe = (float(x) for x in det[d, 3:8])
    rot = float(det[d, 10])
    c, sn = math.cos(rot), math.sin(rot)
    q = [x[None] for x in Q]
    p = [E[:, a:a + 1] for a in range(3)]
    d3 = [b - a for a, b in zip(p, q)]
    sq = (d3[0] ** 2 + d3[1] ** 2 + d3[2] ** 2).sqrt()
    cosang = d3[1] / sq
    att = torch.zeros_like(sq)
    for m, (lo, hi, thick, mu, h0, h1) in enumerate(layers):
        att += 1e5 * (_crossing(p, q, lo, hi) < float(np.float32(0.1))).double()
        pick = (o >= h0) & (o < h1)
        ei, hh = e[pick], hole[o[pick]]
        col = [hh[:, k:k + 1] for k in range(6)]
        chord = _cylinder([E[ei, a:a + 1] for a in range(3)], q, col[0], col[1], col[2], col[3], col[4])
        length = torch.zeros_like(sq).index_add_(0, ei, chord)
        att.index_add_(0, ei, chord * col[5])
        rest = thick / cosang - length
        att += torch.where(rest >= 1e-5, mu * rest, torch.zeros_like(rest))
    pick = o >= H
    ei, k = e[pick], o[pick] - H
    dd = det[k]
    ck, sk = torch.cos(-dd[:, 10:11]), torch.sin(-dd[:, 10:11])

    def frame(x, y, z):
        x, z = x - dd[:, 0:1], z - dd[:, 2:3]
        return x * ck - z * sk, y - dd[:, 1:2], x * sk + z * ck
    half = [0.5 * dd[:, 3 + a:4 + a] for a in range(3)]
    chord = _crossing(frame(*[E[ei, a:a + 1] for a in range(3)]), frame(*q), [-x for x in half], half)
    att.index_add_(0, ei, chord * dd[:, 6:7])
    # crystal d: self attenuation, absorption, solid angle
    cm, sm = math.cos(-rot), math.sin(-rot)
    ex, ey, ez = p[0] - det[d, 0], p[1] - det[d, 1], p[2] - det[d, 2]
    ps, qd = (ex * cm - ez * sm, ey, ex * sm + ez * cm), [x[None] for x in qs]
    size = (w, t, h)
    lo = [((frac[a] - 0.5) * size[a] - 0.5 * size[a] / div[a])[None] for a in range(3)]
    hi = [((frac[a] - 0.5) * size[a] + 0.5 * size[a] / div[a])[None] for a in range(3)]
    l1 = _to_end(ps, qd, [-0.5 * x for x in size], [0.5 * x for x in size])
    l2 = _to_end(ps, qd, lo, hi)
    att += (l1 - l2) * mu_t
    ext = [b + 1000.0 * (b - a) / sq for a, b in zip(ps, qd)]
    labs = _crossing(ps, ext, lo, hi)
    absf = -torch.expm1(-labs * mu_t) * mu_pe / mu_t
    rq = 1.0 / (4 * math.pi * sq ** 3)
    ax, ay, az = t * h / div[2] / div[1], w * h / div[0] / div[2], w * t / div[0] / div[1]
    sa = torch.maximum(torch.maximum(ax * (d3[0] * c - d3[2] * sn).abs(), ay * d3[1].abs()),
                       az * (d3[0] * sn + d3[2] * c).abs()) * rq
    return (torch.exp(-att) * sa * absf).sum(1)


def _kn_integral(cos_t, alpha):
    """Integral of the Klein-Nishina shape times sin from 0, as a function of cos(theta)."""
    b = 1 + alpha

    def prim(p):
        return -(1 + b * b / alpha ** 2) / p - (2 * b / alpha ** 2) * torch.log(p) + p / alpha ** 2 + torch.log(p) + \
            2 / p - 0.5 / p ** 2
    p = 1 + alpha * (1 - cos_t)
    return (prim(p) - prim(torch.ones_like(p))) / alpha


def _kn(th, alpha):
    """Shape times sin and its derivative."""
    c, s = torch.cos(th), torch.sin(th)
    om = 1 - c
    p = 1 + alpha * om
    g = (1 + c * c) / p ** 2 + alpha ** 2 * om * om / p ** 3
    gp = 2 * c / p ** 2 + 2 * alpha * (1 + c * c) / p ** 3 - 2 * alpha ** 2 * om / p ** 3 + \
        3 * alpha ** 3 * om * om / p ** 4
    return g * s, c * g - s * s * gp


def _scatter_exact(geo, seed, case):
    det, hole, _ = _tables(geo)
    D = det.shape[0]
    v0, nv, parts = case["vox"], case["voxs"], case["parts"]
    I = _voxels(geo, 0.0, v0, nv)
    pe = _plain_pe(geo, seed, v0, nv)[:, v0:v0 + nv].double()
    lo, hi, e0 = (float(geo.physics[k]) for k in (5, 6, 7))
    alpha, step = e0 / 511.0, float(np.float32(0.01))
    th = torch.arange(315, dtype=torch.float64) * step
    integ = float((_kn(th, alpha)[0] * step).sum())
    n0 = geo.n_holes_layer0
    points = torch.cat([det[:, :3], torch.stack([hole[:n0, 0], 0.5 * (hole[:n0, 1] + hole[:n0, 2]), hole[:n0, 3]], 1)])
    vr = float(np.float32(0.1))
    toI = points[D:, None] - I[None]
    lih = toI.norm(dim=2)
    sa = (vr * vr * math.pi + (hole[:n0, 2] - hole[:n0, 1])[:, None] * vr) / (4 * math.pi * lih ** 3) * toI[..., 1].abs()
    w_hole = sa / float(geo.collimator[15]) * float(geo.collimator[17])
    s0, s1 = (0 if parts & 1 else D), (D + n0 if parts & 2 else D)
    S = points[s0:s1]
    out = torch.zeros((case["dets"], nv), dtype=torch.float64, device="cuda")
    A = S[:, None] - I[None]                       # voxel -> scatter point
    la = A.norm(dim=2)
    for d in range(case["det"], case["det"] + case["dets"]):
        P, size, (mu_pe, mu_c, eres) = det[d, :3], det[d, 3:6], (float(x) for x in det[d, 7:10])
        weight = (torch.cat([pe * (mu_c / mu_pe), w_hole]))[s0:s1].clone()
        if parts & 1:
            weight[d] = 0
        B = P - S
        lsd = B.norm(dim=1)
        cosc = ((A * B[:, None]).sum(2) / (la * lsd[:, None])).clamp(-1, 1)
        cone = torch.acos(cosc)
        r = 1 + alpha * (1 - cosc)
        es = e0 / r
        res = eres * (1 / r).sqrt()
        inside = (es * (1 + 2 * res / 2.35482) > lo) & (es * (1 - 2 * res / 2.35482) < hi)
        sig = res / 2.35482 * es * math.sqrt(2.0)
        pwin = 0.5 * (torch.erf((hi - es) / sig) - torch.erf((lo - es) / sig))
        rdet = 0.5 * float(size.norm())
        x = rdet / 2 / lsd[:, None] / torch.sin(cone)
        phi = torch.where(x >= 1, torch.full_like(x, 2 * math.pi), 4 * torch.asin(x.clamp(max=1)))
        # the crystals are not rotated: the crystal frame is a shift
        cmin, cmax = torch.full_like(la, 2.0), torch.full_like(la, -2.0)
        for k in range(8):
            corner = P + torch.tensor([(k & 1) - 0.5, (k >> 1 & 1) - 0.5, (k >> 2) - 0.5], dtype=torch.float64,
                                      device="cuda") * size
            b = corner - S
            ck = ((A * b[:, None]).sum(2) / (la * b.norm(dim=1)[:, None])).clamp(-1, 1)
            cmin, cmax = torch.minimum(cmin, ck), torch.maximum(cmax, ck)
        tmin, tmax = torch.acos(cmax), torch.acos(cmin)
        p = [I[None, :, a] - P[a] for a in range(3)]
        q = [S[:, a:a + 1] - P[a] + 1000.0 * A[..., a] / la for a in range(3)]
        half = [0.5 * float(x) for x in size]
        through = _crossing(p, q, [-x for x in half], half) > EPS
        tmin = torch.where(through, torch.zeros_like(tmin), tmin)
        n = torch.floor((tmax - tmin) / step)
        tb = tmin + n * step
        Fa, Pa = _kn(tmin, alpha)
        Fb, Pb = _kn(tb, alpha)
        ratio = (_kn_integral(torch.cos(tb), alpha) - _kn_integral(torch.cos(tmin), alpha) + 0.5 * step * (Fa + Fb) +
                 step * step / 12 * (Pb - Pa)) / integ
        # crystals on the way
        pa = [S[:, a:a + 1] - det[None, :, a] for a in range(3)]
        pb = [(P[a] - det[:, a])[None] for a in range(3)]
        hs = [0.5 * det[None, :, 3 + a] for a in range(3)]
        chord = _crossing([x.expand(S.shape[0], D) for x in pa], [x.expand(S.shape[0], D) for x in pb],
                          [-x for x in hs], hs)
        chord[:, d] = 0
        if parts & 1:
            chord[torch.arange(D, device="cuda"), torch.arange(D, device="cuda")] = 0
        chord = torch.nan_to_num(chord)
        lpe, lc = chord @ det[:, 7], chord @ det[:, 8]
        ext = [-1000.0 * (S[:, a] - P[a]) / lsd for a in range(3)]
        labs = torch.nan_to_num(_crossing([S[:, a] - P[a] for a in range(3)], ext, [-x for x in half], half))
        mpe = mu_pe * r ** 3
        mt = mpe + mu_c * r
        item = weight * phi / 2 / math.pi * ratio * pwin * torch.exp(-(lpe[:, None] * r ** 3 + lc[:, None] * r)) * \
            -torch.expm1(-labs[:, None] * mt) * mpe / mt
        out[d - case["det"]] = torch.where(inside & (weight != 0), item, torch.zeros_like(item)).sum(0)
    return out


def exact(case, seed):
    path = case["path"]
    if path in ("grid", "gradient"):       # no plain form that ends in seconds
        return None
    if path == "batch":
        if case["designs"] * case["dets"] * case["voxs"] > 300000:
            return None
        designs = geometry.config4(case["designs"])
        return [_pe_exact(_varied(g, seed, k + 1), float((7 * k) % g.n_rot), case["det"], case["dets"], case["vox"],
                          case["voxs"]) for k, g in enumerate(designs)]
    geo = _system(case, seed)
    if path == "host":
        if geo.n_det * geo.n_vox > 400000:
            return None
        return _pe_exact(geo, 0.0, 0, geo.n_det, 0, geo.n_vox)
    if path == "projector":
        x, _ = _activity(case, seed)
        on = x.nonzero().flatten()
        A = _pe_exact(geo, 0.0, case["det"], case["dets"], 0, 0, voxels=on)
        return {"p": A @ x[on].double(), "q": None}
    if path == "scatter":
        if case["dets"] * case["voxs"] > 1000000:
            return None
        return {"crystal": None, "collimator": None, "scatter": _scatter_exact(geo, seed, case)}
    div, sub = (_ints(case["div"]), _ints(case["sub"])) if path == "sampled" else ((8, 16, 8), (1, 1, 1))
    if case["dets"] * case["voxs"] * math.prod(div) * math.prod(sub) > 4e8:
        return None
    return _pe_exact(geo, float(case["rot"]), case["det"], case["dets"], case["vox"], case["voxs"], div, sub)
