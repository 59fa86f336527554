"""Performance cases of the framework: the calls its users make, over the range of sizes they make them at.

A case is a dict with a "kind" and the sizes of one call.  The kinds:

fan_fbp     fan weighting -> ramp filter -> fan backprojection of a batch of sinograms, through the functions
            of ``torch_ctrecon`` (the reconstruction of measured fan-beam slices; float64 for small problems,
            where users check gradients and reference results)
fan_train   the same chain with a gradient back to the sinogram (a network that works on sinograms)
par_fbp     parallel projection -> ramp filter -> parallel backprojection (the headline chain)
par_step    one step of iterative reconstruction, x - lr * A^T (A x - y), gradient through autograd
lowp_fbp    large slices stored in 16 bits (or 32): tensor-core filter with fused weighting -> fan backprojection
fan_batch   a plan of fan slices that all differ in image size, views and channels
single_view one backprojected image per view (input of per-view networks)
raycast     the ray-casting projector (sub-pixel sampling inside the field of view)
disdriven   the distance-driven projector and its gradient kernel
helical     rebinning of a helical scan to fan sinograms, 360LI or 180LI
"""
import math

import numpy as np
import torch

from ct_recon_extensions_gb300 import torch_ctrecon as tc
from ct_recon_extensions_gb300.batch import FanFBPBatch

DSO, DSD = 595.0, 1085.6  # source to centre and to detector, mm
FOV = 256.0               # image side, mm
ARC = 1.2858 * 736        # detector arc of a fan scan, mm
DTYPE = {"f32": torch.float32, "f64": torch.float64, "bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    return [
        # a small slice: latency and launches of a three-operator chain
        {"name": "fan_fbp_128", "kind": "fan_fbp", "n": 128, "na": 180, "ns": 185, "batch": 1, "dtype": "f32"},
        # the ordinary clinical fan slice (720 views x 736 channels -> 512 x 512), forward and backward
        {"name": "fan_train_512", "kind": "fan_train", "n": 512, "na": 720, "ns": 736, "batch": 1},
        # the headline chain: 512 x 512, 720 views x 729 bins
        {"name": "par_fbp_512", "kind": "par_fbp", "n": 512, "na": 720, "ns": 729, "batch": 1},
        # iterative reconstruction of one slice
        {"name": "par_step_512x1", "kind": "par_step", "n": 512, "na": 720, "ns": 729, "batch": 1},
        # iterative reconstruction of a stack of slices
        {"name": "par_step_512x16", "kind": "par_step", "n": 512, "na": 720, "ns": 729, "batch": 16},
        # a large slice stored in 16 bits
        {"name": "lowp_fbp_2048", "kind": "lowp_fbp", "n": 2048, "na": 2304, "ns": 1472, "dtype": "bf16", "splits": 3},
        # uneven slices reconstructed together
        {"name": "fan_batch_16", "kind": "fan_batch", "items": 16, "low": 256, "high": 1024, "sizes": 3000},
        # per-view images at the headline size (755 MB out)
        {"name": "single_view_512", "kind": "single_view", "n": 512, "na": 720, "ns": 729, "batch": 1},
        # the other two projectors of the reference's operator
        {"name": "raycast_512", "kind": "raycast", "n": 512, "na": 720, "ns": 729, "batch": 1, "step": 0.125},
        {"name": "disdriven_512", "kind": "disdriven", "n": 512, "na": 720, "ns": 729, "batch": 1},
        # a clinical helical scan: 64 rows, 1152 views per rotation, 128 slices
        {"name": "helical_360", "kind": "helical", "method": "360", "ns": 736, "nt": 64, "vpr": 1152, "nz": 128,
         "thickness": 1.0},
        {"name": "helical_180", "kind": "helical", "method": "180", "ns": 736, "nt": 64, "vpr": 1152, "nz": 128,
         "thickness": 1.0},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["fan_fbp", "fan_train", "par_fbp", "par_step", "lowp_fbp", "fan_batch", "single_view",
                       "raycast", "disdriven", "helical"])
    n = _log(rng, 64, 512)
    na = min(1024, max(24, int(n * rng.uniform(0.8, 1.8))))
    ns = int(n * rng.uniform(1.0, 1.5)) + rng.randint(0, 3)
    if kind in ("fan_fbp", "fan_train"):
        c = {"n": n, "na": na, "ns": ns, "batch": rng.randint(1, 4)}
        if kind == "fan_fbp":
            c["dtype"] = "f64" if n <= 128 and rng.random() < 0.5 else "f32"
    elif kind == "par_fbp":
        c = {"n": n, "na": na, "ns": ns, "batch": rng.randint(1, 4)}
    elif kind == "par_step":
        c = {"n": n, "na": na, "ns": ns, "batch": _log(rng, 1, 16) if n * n * na <= 512 * 512 * 720 else 1}
    elif kind == "lowp_fbp":
        c = {"n": _log(rng, 512, 2048), "na": _log(rng, 512, 2304), "ns": _log(rng, 512, 1472),
             "dtype": rng.choice(["bf16", "f16", "f32"]), "splits": rng.choice([2, 3, 3])}
    elif kind == "fan_batch":
        c = {"items": _log(rng, 2, 16), "low": 128, "high": rng.randint(256, 768), "sizes": rng.randint(0, 10 ** 6)}
    elif kind == "single_view":
        na = min(na, 720)
        c = {"n": n, "na": na, "ns": ns, "batch": 1 if n > 256 else rng.randint(1, 4)}
    elif kind == "raycast":
        c = {"n": n, "na": min(na, 720), "ns": ns, "batch": 1, "step": rng.choice([0.125, 0.25, 0.5])}
    elif kind == "disdriven":
        c = {"n": n, "na": na, "ns": ns, "batch": rng.randint(1, 2) if n < 400 else 1}
    else:
        vpr = rng.randint(45, 144) * 8
        c = {"method": rng.choice(["360", "180"]), "ns": rng.randint(256, 736), "nt": rng.choice([16, 32, 64]),
             "vpr": vpr, "nz": _log(rng, 8, 96), "thickness": rng.choice([0.75, 1.0, 2.5])}
    return {"kind": kind, **c}


# ---- geometry --------------------------------------------------------------

def _fan(c):
    """Fan geometry of a case: full rotation, constant field of view and fan angle."""
    d = FOV / c["n"]
    return dict(n=c["n"], na=c["na"], ns=c["ns"], d=d, ds=ARC / c["ns"], orbit=2 * math.pi / c["na"])


def _par(c):
    """Parallel geometry: half a rotation, bins of a pixel's width."""
    d = FOV / c["n"]
    return dict(n=c["n"], na=c["na"], ns=c["ns"], d=d, ds=d, orbit=math.pi / c["na"])


def _par_kw(g):
    return dict(img_shape=(g["n"], g["n"]), img_space=(g["d"], g["d"]), proj_shape=(g["na"], g["ns"]),
                channel_space=g["ds"], orbit=g["orbit"])


def _fan_kw(g):
    return dict(_par_kw(g), dso=DSO, dsd=DSD)


def _batch_geoms(c):
    """The items of a fan_batch case, from the case alone."""
    rng = np.random.default_rng(c["sizes"])
    out = []
    for _ in range(c["items"]):
        n = int(rng.integers(c["low"], c["high"] + 1))
        na = int(rng.integers(360, max(361, int(2.25 * c["high"]))))
        ns = int(rng.integers(max(256, c["high"] // 2), max(257, c["high"] + 1)))
        out.append(dict(ns=ns, na=na, ds=ARC / ns, orbit=2 * math.pi / na, offset_s=0.0, orbit_start=0.0, nx=n, ny=n,
                        dx=FOV / n, dy=FOV / n, offset_x=0.0, offset_y=0.0, dso=DSO, dsd=DSD, fov=-1.0))
    return out


def _helical(c):
    """A scan of pitch 1: slices nine views apart, views enough around every slice."""
    vpr, nt, nz = c["vpr"], c["nt"], c["nz"]
    cm = nt * DSO / DSD / vpr
    step = 9
    c0 = vpr + 8
    na = c0 + step * (nz - 1) + vpr + 8
    return dict(ns=c["ns"], nt=nt, na=na, ds=ARC / c["ns"], dt=1.0, offset_s=1.25, offset_t=0.0, orbit_start=0.0,
                orbit=2 * math.pi / vpr, couch_begin=0.0, couch_mov=cm, view_per_rot=vpr, nz=nz, dz=step * cm,
                z0=c0 * cm + 0.1 * cm, thickness=c["thickness"], dso=DSO, dsd=DSD)


# ---- inputs ----------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _ellipses(gen, batch, n=10):
    """Random ellipse phantoms: centre, semi-axes, orientation and attenuation (1/mm) of n ellipses an item."""
    u = torch.rand(6, batch, n, 1, 1, generator=gen, device="cuda", dtype=torch.float32)
    r, t = 100.0 * u[0].sqrt(), 2 * math.pi * u[1]
    return (r * t.cos(), r * t.sin(), 5 + 55 * u[2], 5 + 55 * u[3], math.pi * u[4], 0.01 + 0.02 * u[5])


def _images(gen, batch, n):
    d = FOV / n
    p = (torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1) / 2) * d
    x, y = p[None, :], -p[:, None]
    e = _ellipses(gen, batch)
    out = torch.zeros(batch, n, n, device="cuda")
    for i in range(10):
        cx, cy, a, b, phi, mu = (v[:, i] for v in e)
        u = (x - cx) * phi.cos() + (y - cy) * phi.sin()
        v = -(x - cx) * phi.sin() + (y - cy) * phi.cos()
        out += mu * ((u / a) ** 2 + (v / b) ** 2 <= 1)
    return out


def _sinograms(gen, batch, theta, s):
    """Line integrals of random phantoms along x cos(theta) + y sin(theta) = s, with the noise of a scan."""
    theta, s = (v.to(torch.float32) for v in torch.broadcast_tensors(theta, s))
    e = _ellipses(gen, batch)
    out = torch.zeros((batch,) + tuple(theta.shape), device="cuda")
    for i in range(10):
        cx, cy, a, b, phi, mu = (v[:, i] for v in e)
        r2 = (a * (theta - phi).cos()) ** 2 + (b * (theta - phi).sin()) ** 2
        q = s - (cx * theta.cos() + cy * theta.sin())
        out += 2 * mu * a * b * (r2 - q * q).clamp_(min=0).sqrt_() / r2
    out += 0.01 * torch.randn(out.shape, generator=gen, device="cuda")
    return out


def _fan_sinograms(gen, batch, g):
    beta = torch.arange(g["na"], device="cuda", dtype=torch.float64)[:, None] * g["orbit"]
    gamma = (torch.arange(g["ns"], device="cuda", dtype=torch.float64) - (g["ns"] - 1) / 2) * g["ds"] / DSD
    return _sinograms(gen, batch, beta + gamma, DSO * gamma.sin())


def _par_sinograms(gen, batch, g):
    theta = torch.arange(g["na"], device="cuda", dtype=torch.float64)[:, None] * g["orbit"]
    s = (torch.arange(g["ns"], device="cuda", dtype=torch.float64) - (g["ns"] - 1) / 2) * g["ds"]
    return _sinograms(gen, batch, theta, s)


def _inputs(c, seed):
    gen, kind = _gen(seed), c["kind"]
    if kind in ("fan_fbp", "fan_train"):
        g = _fan(c)
        x = {"sino": _fan_sinograms(gen, c["batch"], g).to(DTYPE[c.get("dtype", "f32")])}
        if kind == "fan_train":
            x["grad"] = _images(gen, c["batch"], g["n"]) + 0.01
        return x
    if kind == "lowp_fbp":
        return {"sino": _fan_sinograms(gen, 1, _fan(c)).to(DTYPE[c["dtype"]])}
    if kind == "fan_batch":
        return {"sinos": [_fan_sinograms(gen, 1, g)[0] for g in _batch_geoms(c)]}
    if kind in ("par_fbp", "raycast"):
        return {"img": _images(gen, c["batch"], c["n"])}
    if kind == "par_step":
        return {"img": _images(gen, c["batch"], c["n"]), "sino": _par_sinograms(gen, c["batch"], _par(c))}
    if kind == "disdriven":
        return {"img": _images(gen, c["batch"], c["n"]), "sino": _par_sinograms(gen, c["batch"], _par(c))}
    if kind == "single_view":
        return {"sino": _par_sinograms(gen, c["batch"], _par(c))}
    h = _helical(c)
    base = _fan_sinograms(gen, 1, dict(na=h["na"], ns=h["ns"], ds=h["ds"], orbit=h["orbit"]))[0]
    rows = 1 + 0.2 * torch.rand(h["nt"], 1, generator=gen, device="cuda")
    x = base[:, None, :] * rows
    x += 0.01 * torch.randn(x.shape, generator=gen, device="cuda")
    return {"proj": x}


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"kind": kind, "in": _inputs(c, seed), "case": c}
    if kind in ("fan_fbp", "fan_train", "lowp_fbp"):
        s["g"] = g = _fan(c)
        s["kw"] = _fan_kw(g)
        if kind == "lowp_fbp":
            w = tc.FanWeightingOp(g["ns"], g["na"], g["ds"], 0.0, DSO, DSD, 1)
            s["filter"] = tc.RampFilterTCOp(g["ns"], g["na"], g["ds"], DSD, 1, weighting=w, splits=c["splits"])
    elif kind == "fan_batch":
        s["plan"] = FanFBPBatch(_batch_geoms(c))
    elif kind == "helical":
        s["op"] = tc.HelicalInterpolationOp(**_helical(c), method=c["method"])
    else:
        s["g"] = g = _par(c)
        s["kw"] = _par_kw(g)
        if kind == "raycast":
            s["op"] = tc.ParallelProjection2DOp(g["ns"], g["na"], g["ds"], g["orbit"], 0.0, 0.0, g["n"], g["n"],
                                                g["d"], g["d"], 0.0, 0.0, FOV / 2, "raycasting", c["step"])
    return s


# ---- one pass --------------------------------------------------------------

def _fan_chain(sino, g, kw):
    w = tc.fan_weighting(sino, (g["na"], g["ns"]), g["ds"], 0, DSO, DSD, "fan")
    return tc.fan_backprojection_2d(tc.ramp_filter(w, g["ns"], g["na"], g["ds"], DSD, "fan"), **kw)


def run(state):
    kind, x = state["kind"], state["in"]
    if kind == "fan_fbp":
        return _fan_chain(x["sino"], state["g"], state["kw"])
    if kind == "fan_train":
        sino = x["sino"].detach().requires_grad_(True)
        img = _fan_chain(sino, state["g"], state["kw"])
        grad, = torch.autograd.grad(img, sino, x["grad"])
        return {"image": img.detach(), "grad": grad}
    if kind == "par_fbp":
        g, kw = state["g"], state["kw"]
        sino = tc.parallel_projection_2d(x["img"], **kw)
        return {"sino": sino, "image": tc.parallel_backprojection_2d(
            tc.ramp_filter(sino, g["ns"], g["na"], g["ds"], -1, "par"), **kw)}
    if kind == "par_step":
        img = x["img"].detach().requires_grad_(True)
        proj = tc.parallel_projection_2d(img, **state["kw"])
        grad, = torch.autograd.grad(proj, img, proj.detach() - x["sino"])
        return {"proj": proj.detach(), "grad": grad, "image": torch.add(x["img"], grad, alpha=-LR)}
    if kind == "lowp_fbp":
        sino = state["filter"].forward(x["sino"])
        return {"sino": sino, "image": tc.fan_backprojection_2d(sino, **state["kw"])}
    if kind == "fan_batch":
        return state["plan"].run(x["sinos"])
    if kind == "single_view":
        return tc.parallel_single_view_bp_2d(x["sino"], **state["kw"])
    if kind == "raycast":
        return state["op"].forward(x["img"])
    if kind == "disdriven":
        kw = state["kw"]
        return {"proj": tc.parallel_projection_2d(x["img"], method="disdriven", **kw),
                "grad": tc.parallel_projection_2d_grad(x["sino"], method="disdriven", **kw)}
    return state["op"].forward(x["proj"])


LR = 1e-6  # step of par_step


# ---- the work of one pass --------------------------------------------------

# operations of one pixel-view update, ray sample or filter product
FAN_UPDATE, PAR_UPDATE, RAY_SAMPLE, TAP = 32, 9, 6, 2


def work(case):
    c, kind = case, case["kind"]
    if kind == "helical":
        h = _helical(c)
        out = h["nz"] * h["view_per_rot"] * h["ns"]
        rows = c["thickness"] * DSD / DSO  # detector rows of a slab
        # input rows that some slice covers: the couch path of the slices and two slabs' width, over the views
        span = min(h["nt"], (h["nz"] - 1) * 9 * h["couch_mov"] * DSD / DSO + 2 * rows)
        used = min(h["na"], 2 * h["view_per_rot"] if c["method"] == "360" else h["view_per_rot"]) * span
        return {"bytes": 4 * (out + used * h["ns"]), "flops": out * (2 * rows + 6)}
    if kind == "fan_batch":
        w = {"bytes": 0, "flops": 0}
        for g in _batch_geoms(c):
            w["bytes"] += 4 * (g["na"] * g["ns"] + g["nx"] * g["ny"])
            w["flops"] += FAN_UPDATE * g["na"] * g["nx"] * g["ny"] + TAP * g["na"] * g["ns"] * g["ns"] // 2
        return w
    n, na, ns, b = c["n"], c["na"], c["ns"], c.get("batch", 1)
    img, sino = n * n, na * ns
    size = {"f64": 8, "bf16": 2, "f16": 2}.get(c.get("dtype"), 4)
    ramp = TAP * sino * ns // 2
    if kind in ("fan_fbp", "lowp_fbp"):
        more = 4 * sino if kind == "lowp_fbp" else 0
        return {"bytes": b * (size * sino + more + (8 if size == 8 else 4) * img),
                "flops": b * (FAN_UPDATE * img * na + ramp)}
    if kind == "fan_train":
        return {"bytes": 4 * b * (2 * sino + 2 * img), "flops": 2 * b * (FAN_UPDATE * img * na + ramp)}
    if kind == "par_fbp":
        return {"bytes": 4 * b * (2 * img + sino), "flops": b * ((PAR_UPDATE + RAY_SAMPLE) * img * na + ramp)}
    if kind == "par_step":
        return {"bytes": 4 * b * (3 * img + 2 * sino), "flops": b * 2 * RAY_SAMPLE * img * na}
    if kind == "single_view":
        return {"bytes": 4 * b * (sino + img * na), "flops": 3 * b * img * na}
    if kind == "raycast":
        chord = math.pi / 4 * n / c["step"]  # mean samples of a ray that meets the field of view
        return {"bytes": 4 * b * (img + sino), "flops": 10 * b * na * min(ns, n) * chord}
    return {"bytes": 8 * b * (img + sino), "flops": 12 * b * 2 * img * na}


# ---- the same in 64 bits ---------------------------------------------------

F64 = dict(device="cuda", dtype=torch.float64)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _sums(start, step, n):
    """start, start + step, start + 2 step, ... as running sums."""
    return np.add.accumulate(np.concatenate([[start], np.full(n - 1, step)]))


def _grid(n, d):
    return _dev(_sums(-(n - 1) / 2 * d, d, n)), _dev(_sums((n - 1) / 2 * d, -d, n))


def _taps(ns, ds, fan):
    k = torch.arange(-(ns - 1), ns, **F64)
    den = (math.pi * DSD * torch.sin(k * ds / DSD)) ** 2 if fan else (math.pi * ds * k) ** 2
    h = torch.where(k.remainder(2) == 1, -1 / den, torch.zeros_like(k))
    h[ns - 1] = 0.25 / ds ** 2
    return h


def _ramp64(x, ns, ds, fan):
    i = torch.arange(ns, device="cuda")
    return x @ (_taps(ns, ds, fan)[i[:, None] - i[None, :] + ns - 1] * ds)


def _weight64(x, g):
    s = g["ds"] * (torch.arange(g["ns"], **F64) - (g["ns"] - 1) / 2)
    return x * (DSO * torch.cos(s / DSD).abs() / DSD)


def _lerp_index(s, ns):
    on = (s >= 0) & (s <= ns - 1)
    s = torch.where(on, s, torch.zeros_like(s))
    i = s.floor()
    return on, i.long(), s.ceil().long(), s - i


def _fan_taps(g, ia, angle, x, y):
    sb, cb = math.sin(angle[ia]), math.cos(angle[ia])
    r, q = x * cb + y * sb, DSO + x * sb - y * cb
    on, i1, i2, u = _lerp_index(torch.atan2(r, q) * (DSD / g["ds"]) + (g["ns"] - 1) / 2, g["ns"])
    return i1, i2, u, torch.where(on, DSD * DSD / (q * q + r * r), torch.zeros_like(u))


def _fan_bp64(p, g):
    xs, ys = _grid(g["n"], g["d"])
    x, y = xs[None, :], ys[:, None]
    angle = _sums(0.0, g["orbit"], g["na"])
    out = torch.zeros(p.shape[0], g["n"], g["n"], **F64)
    for ia in range(g["na"]):
        i1, i2, u, w = _fan_taps(g, ia, angle, x, y)
        out += ((1 - u) * p[:, ia][:, i1] + u * p[:, ia][:, i2]) * w
    return out * (g["orbit"] / round(g["na"] * g["orbit"] / math.pi))


def _fan_bp64_t(img, g):
    xs, ys = _grid(g["n"], g["d"])
    x, y = xs[None, :], ys[:, None]
    angle = _sums(0.0, g["orbit"], g["na"])
    out = torch.zeros(img.shape[0], g["na"], g["ns"], **F64)
    for ia in range(g["na"]):
        i1, i2, u, w = _fan_taps(g, ia, angle, x, y)
        for b in range(img.shape[0]):
            out[b, ia].index_add_(0, i1.reshape(-1), (img[b] * w * (1 - u)).reshape(-1))
            out[b, ia].index_add_(0, i2.reshape(-1), (img[b] * w * u).reshape(-1))
    return out * (g["orbit"] / round(g["na"] * g["orbit"] / math.pi))


def _par_s(g, ia, angle, xs, ys):
    return (xs[None, :] * math.cos(angle[ia]) + ys[:, None] * math.sin(angle[ia])) / g["ds"] + (g["ns"] - 1) / 2


def _par_bp64(p, g):
    xs, ys = _grid(g["n"], g["d"])
    angle = _sums(0.0, g["orbit"], g["na"])
    out = torch.zeros(p.shape[0], g["n"], g["n"], **F64)
    for ia in range(g["na"]):
        on, i1, i2, u = _lerp_index(_par_s(g, ia, angle, xs, ys), g["ns"])
        out += ((1 - u) * p[:, ia][:, i1] + u * p[:, ia][:, i2]) * on
    return out * g["orbit"]


def _single64(p, g):
    xs, ys = _grid(g["n"], g["d"])
    angle = _sums(0.0, g["orbit"], g["na"])
    out = torch.empty(p.shape[0], g["n"], g["n"], g["na"], **F64)
    for ia in range(g["na"]):
        on, i1, i2, u = _lerp_index(_par_s(g, ia, angle, xs, ys), g["ns"])
        out[..., ia] = ((1 - u) * p[:, ia][:, i1] + u * p[:, ia][:, i2]) * on
    return out


def _along_x(a):
    return not (math.pi / 4 <= a < 3 * math.pi / 4 or 5 * math.pi / 4 <= a < 7 * math.pi / 4)


def _ray_starts(g, angle):
    """(start of every channel on the first line, step per line, length of a line's step, marched along y) of a view."""
    n, ns, d, ds = g["n"], g["ns"], g["d"], g["ds"]
    c, cents = (n - 1) / 2, (ns - 1) / 2
    sa, ca = math.sin(angle), math.cos(angle)
    if _along_x(angle):
        step, chan, length = sa / ca, ds / (ca * d), abs(d / ca)
    else:
        step, chan, length = ca / sa, -ds / (sa * d), abs(d / sa)
    return _sums(c - c * step - cents * chan, chan, ns), step, chan, length, _along_x(angle)


def _par_fp64(img, g):
    n = g["n"]
    angle = _sums(0.0, g["orbit"], g["na"])
    flat = img.reshape(img.shape[0], -1), img.transpose(1, 2).reshape(img.shape[0], -1)
    line = torch.arange(n, device="cuda")[:, None] * n
    out = torch.empty(img.shape[0], g["na"], g["ns"], **F64)
    for ia in range(g["na"]):
        start, step, _, length, ux = _ray_starts(g, angle[ia])
        pos = np.full((n, g["ns"]), step)
        pos[0] = start
        on, i1, i2, u = _lerp_index(_dev(np.add.accumulate(pos, axis=0)), n)
        f = flat[0 if ux else 1]
        for b in range(img.shape[0]):
            out[b, ia] = (((1 - u) * f[b][i1 + line] + u * f[b][i2 + line]) * on).sum(0) * length
    return out


def _pixel_footprints(g, angle):
    """Channel of every pixel in a view and the ends of its footprint, on the image's own axes."""
    n, d, ds = g["n"], g["d"], g["ds"]
    c, cents = (n - 1) / 2, (g["ns"] - 1) / 2
    sa, ca = math.sin(angle), math.cos(angle)
    ux = _along_x(angle)
    a, b = (d * ca / ds, -d * sa / ds) if ux else (-d * sa / ds, d * ca / ds)
    mid = _dev(_sums(cents - c * a - c * b, b, n))[:, None] + a * torch.arange(n, **F64)[None, :]
    left, right = mid - a, mid + a
    left[:, 0], right[:, -1] = mid[:, 0], mid[:, -1]
    turn = (lambda v: v) if ux else (lambda v: v.t())
    return (turn(mid), turn(torch.minimum(left, right)), turn(torch.maximum(left, right)), a,
            abs(d / ca) if ux else abs(d / sa))


def _par_fp64_t(p, g):
    ns = g["ns"]
    angle = _sums(0.0, g["orbit"], g["na"])
    out = torch.zeros(p.shape[0], g["n"], g["n"], **F64)
    for ia in range(g["na"]):
        mid, left, right, a, length = _pixel_footprints(g, angle[ia])
        lo, hi = left.ceil().clamp(min=0), right.floor().clamp(max=ns - 1)
        for k in range(int(2 * abs(a)) + 2):
            i = lo + k
            w = (1 - (mid - i).abs() / abs(a)) * (i <= hi) * length
            i = i.clamp(0, ns - 1).long()
            out += w * p[:, ia][:, i]
    return out


def _raycast64(img, g, step):
    n, fov = g["n"], FOV / 2
    angle = _sums(0.0, g["orbit"], g["na"])
    sa, ca = _dev(np.sin(angle))[:, None], _dev(np.cos(angle))[:, None]
    s = _dev(_sums(-(g["ns"] - 1) / 2 * g["ds"], g["ds"], g["ns"]))[None, :]
    h2 = fov * fov - s * s
    h = h2.clamp(min=0).sqrt()
    c = (n - 1) / 2
    x1, y1 = (s * ca - h * sa) / g["d"] + c, -(s * sa + h * ca) / g["d"] + c
    x2, y2 = (s * ca + h * sa) / g["d"] + c, -(s * sa - h * ca) / g["d"] + c
    sx, sy = step * sa, step * ca
    count = torch.where(sa > 1.0 / 1.414, (x2 - x1) / sx, (y2 - y1) / sy).trunc() * (h2 > 0)
    x, y = x1.clone(), y1.clone()
    out = torch.zeros(img.shape[0], g["na"], g["ns"], **F64)
    f = img.reshape(img.shape[0], -1)
    for k in range(int(count.max().item())):
        on = (x >= 0) & (x <= n - 1) & (y >= 0) & (y <= n - 1) & (k < count)
        xc, yc = torch.where(on, x, 0.0), torch.where(on, y, 0.0)
        i, j = xc.floor(), yc.floor()
        u, v = xc - i, yc - j
        i, j, i2, j2 = i.long(), j.long() * n, xc.ceil().long(), yc.ceil().long() * n
        for b in range(img.shape[0]):
            p = f[b]
            out[b] += ((1 - v) * ((1 - u) * p[j + i] + u * p[j + i2]) + v * ((1 - u) * p[j2 + i] + u * p[j2 + i2])) * on
        x += sx
        y += sy
    return out * (step * g["d"])


def _disdriven64(img, g):
    n, na, ns = g["n"], g["na"], g["ns"]
    angle = _sums(0.0, g["orbit"], na)
    rays = [_ray_starts(g, a) for a in angle]
    out = torch.zeros(img.shape[0], na, ns, **F64)
    for ux in (True, False):
        views = [i for i in range(na) if rays[i][4] is ux]
        if not views:
            continue
        at = torch.tensor(views, device="cuda")
        mid = _dev(np.stack([rays[i][0] for i in views]))
        half = _dev(np.array([abs(rays[i][2]) / 2 for i in views]))[:, None]
        step = _dev(np.array([rays[i][1] for i in views]))[:, None]
        length = _dev(np.array([rays[i][3] for i in views]))[:, None]
        src = (img if ux else img.transpose(1, 2)).contiguous()
        left, right = mid - half, mid + half
        width = int(2 * half.max().item()) + 2
        total = torch.zeros(img.shape[0], len(views), ns, **F64)
        for line in range(n):
            first = left.floor()
            sums = torch.zeros_like(total)
            lens = torch.zeros_like(left)
            for k in range(width):
                i = first + k
                on = (first >= 0) & (i < right.ceil()) & (i < n - 1)
                part = (torch.minimum(i + 1, right) - torch.maximum(i, left)) * on
                i = i.clamp(0, n - 2).long()
                row = src[:, line]
                sums += part * (row[:, i] + row[:, i + 1]) / 2
                lens += part
            total += torch.where(lens > 0, sums / lens, torch.zeros_like(sums))
            left, right = left + step, right + step
        out[:, at] = total * length
    return out


def _disdriven64_grad(p, g):
    na, ns = g["na"], g["ns"]
    angle = _sums(0.0, g["orbit"], na)
    pad = torch.cat([p.reshape(p.shape[0], -1), torch.zeros(p.shape[0], 1, **F64)], 1)
    out = torch.zeros(p.shape[0], g["n"], g["n"], **F64)
    for ia in range(na):
        _, left, right, a, length = _pixel_footprints(g, angle[ia])
        c0, c1 = (left - 0.5).ceil(), (right + 0.5).floor()
        for k in range(int(2 * abs(a)) + 3):
            i = c0 + k
            part = (torch.minimum(i + 0.5, right) - torch.maximum(i - 0.5, left)) * ((c0 >= 0) & (i <= c1)) * length / 2
            out += part * pad[:, (i + ia * ns).clamp(0, na * ns).long()]
    return out


def _heli_rows64(h, zd, cg):
    ct = (h["nt"] - 1) / 2
    top = ct - (zd + h["thickness"] / 2) / DSO * cg * DSD
    bot = ct - (zd - h["thickness"] / 2) / DSO * cg * DSD
    on = (bot >= 0) & (top < h["nt"])
    r0 = top.clamp(min=0).floor()
    r1 = bot.clamp(max=h["nt"]).ceil()
    return on, torch.where(on, r0, 0.0).long(), torch.where(on, r1, 1.0).long()


def _helical64(x, h, method):
    vpr, ns, nt, na = h["view_per_rot"], h["ns"], h["nt"], h["na"]
    run_sum = torch.zeros(na, nt + 1, ns, **F64)
    torch.cumsum(x.to(torch.float64), 1, out=run_sum[:, 1:])
    flat = run_sum.reshape(-1)
    cs = (ns - 1) / 2 + h["offset_s"]
    s = (torch.arange(ns, **F64) - cs) * h["ds"]
    gamma = s / DSD
    cg = torch.cos(gamma)[None, :]
    chan = torch.arange(ns, device="cuda")[None, :]

    def rows(view, r0, r1, c):
        at = view * ((nt + 1) * ns) + c
        return (flat[at + r1 * ns] - flat[at + r0 * ns]) / (r1 - r0)

    out = torch.empty(h["nz"], vpr, ns, **F64)
    z = h["z0"]
    for iz in range(h["nz"]):
        centre = int(math.floor((z - h["couch_begin"]) / h["couch_mov"] + 0.5))
        iv = torch.arange(vpr, device="cuda")[:, None]
        if method == "360":
            lo = centre - vpr
            cur = (lo // vpr + 1) * vpr + iv
            cor = torch.where(cur >= centre, cur - vpr, cur + vpr)
            zd, zd2 = (z - h["couch_begin"] - v.double() * h["couch_mov"] for v in (cur, cor))
            on, r0, r1 = _heli_rows64(h, zd, cg)
            on2, q0, q1 = _heli_rows64(h, zd2, cg)
            a, b = rows(cur, r0, r1, chan), rows(cor, q0, q1, chan)
        else:
            lo = centre - vpr // 2
            hi = lo + vpr - 1
            cur = -(-lo // vpr) * vpr + iv
            cur = torch.where(cur > hi, cur - vpr, cur)
            zd = z - h["couch_begin"] - cur.double() * h["couch_mov"]
            on, r0, r1 = _heli_rows64(h, zd, cg)
            a = rows(cur, r0, r1, chan)
            cv = cur.double() - (math.pi - 2 * gamma[None, :]) / h["orbit"]
            cv = torch.where(cv < lo, cv + vpr, cv)
            cv = torch.where(cv > hi, cv - vpr, cv)
            zd2 = z - h["couch_begin"] - cv * h["couch_mov"]
            on2, q0, q1 = _heli_rows64(h, zd2, cg)
            sc = cs - s / h["ds"]
            off = (sc < 0) | (sc > ns - 1)
            cl, cr = sc.floor().clamp(0, ns - 1).long()[None, :], sc.ceil().clamp(0, ns - 1).long()[None, :]
            v = (sc - sc.floor())[None, :]
            vl, vr = cv.floor().long().clamp(0, na - 1), cv.ceil().long().clamp(0, na - 1)
            u = cv - cv.floor()
            b = ((1 - u) * ((1 - v) * rows(vl, q0, q1, cl) + v * rows(vl, q0, q1, cr))
                 + u * ((1 - v) * rows(vr, q0, q1, cl) + v * rows(vr, q0, q1, cr)))
            alone = on2 & off[None, :]  # mirrored channel off the detector: the measured sample as it is
            a, on, on2 = torch.where(alone & ~on, torch.zeros_like(a), a), on | alone, on2 & ~alone
        both = (zd * b - zd2 * a) / (zd - zd2)
        out[iz] = torch.where(on & on2, both, torch.where(on, a, b))
        z += h["dz"]
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    x = {k: [t.double() for t in v] if isinstance(v, list) else v.double() if kind != "helical" else v
         for k, v in _inputs(c, seed).items()}
    if kind in ("fan_fbp", "fan_train", "lowp_fbp"):
        g = _fan(c)
        sino = _ramp64(_weight64(x["sino"], g), g["ns"], g["ds"], True)
        if kind == "fan_fbp":
            return _fan_bp64(sino, g)
        if kind == "lowp_fbp":
            return {"sino": sino, "image": _fan_bp64(sino, g)}
        grad = _fan_bp64_t(x["grad"], g)
        return {"image": _fan_bp64(sino, g), "grad": _weight64(_ramp64(grad, g["ns"], g["ds"], True), g)}
    if kind == "fan_batch":
        out = []
        for p, q in zip(x["sinos"], _batch_geoms(c)):
            g = dict(n=q["nx"], na=q["na"], ns=q["ns"], d=q["dx"], ds=q["ds"], orbit=q["orbit"])
            out.append(_fan_bp64(_ramp64(_weight64(p[None], g), g["ns"], g["ds"], True), g)[0])
        return out
    if kind == "helical":
        return _helical64(x["proj"], _helical(c), c["method"])
    g = _par(c)
    if kind == "par_fbp":
        sino = _par_fp64(x["img"], g)
        return {"sino": sino, "image": _par_bp64(_ramp64(sino, g["ns"], g["ds"], False), g)}
    if kind == "par_step":
        proj = _par_fp64(x["img"], g)
        grad = _par_fp64_t(proj - x["sino"], g)
        return {"proj": proj, "grad": grad, "image": x["img"] - LR * grad}
    if kind == "single_view":
        return _single64(x["sino"], g)
    if kind == "raycast":
        return _raycast64(x["img"], g, c["step"])
    return {"proj": _disdriven64(x["img"], g), "grad": _disdriven64_grad(x["sino"], g)}
