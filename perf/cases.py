"""Performance cases of the projector: what its users run, over the sizes they run it at.

Every case builds its inputs from a seed (an elliptical body with ellipsoidal inserts per material, 1-keV spectra
with smooth attenuation tables, grid and detector tables, measured projections of another body), keeps the plan
and the tables a program would keep, and times one pass through the public entry points:

  forward   Projector.forward: every view's intensities (the projection of a phantom)
  host      Projector.forward_host: the same from and to host memory, as the drop-in classes use it
  subset    forward_views + backward_views of a few consecutive views (one ordered-subset iteration)
  lines     line_integrals and their adjoint (one step of an algebraic reconstruction)
  train     project() under torch.autograd with the log-intensity loss, and its backward
  fused     LogIntensityLoss (forward + loss + adjoint in one launch) and its backward
  batch     Batch.forward_adjoint over uneven problems

`exact` restates the projection in 64-bit torch: the geometry's FP32 scalars as the plan derives them, everything
after them in FP64 (the texture modes at the FP32 sample coordinates and 8-bit weights they are defined by).
"""
import math
import random

import numpy as np
import torch

from ct_forward_projection_b200 import Batch, Projector
from ct_forward_projection_b200.autograd import LogIntensityLoss, project

DEV = "cuda:0"
I0VAL = 60000.0


def _case(name, kind, n, vox, M, views, U, V, pitch, E, mode="trilinear", grid="none", det=True, skip=False, sub=0,
          items=1, pick=0, sod=1000.0, sdd=1500.0, rot=1):
    nx, ny, nz = n
    vx, vy, vz = vox
    return {"name": name, "kind": kind, "mode": mode, "nx": nx, "ny": ny, "nz": nz, "vx": vx, "vy": vy, "vz": vz,
            "M": M, "views": views, "U": U, "V": V, "pitch": pitch, "E": E, "grid": grid, "det": det, "skip": skip,
            "sub": sub, "items": items, "pick": pick, "sod": sod, "sdd": sdd, "rot": rot}


def listed():
    return [
        # the smallest call: a phantom preview or a calibration scan, a few views of a coarse volume
        _case("forward_small_32", "forward", (32, 32, 32), (1.0, 1.0, 1.0), 2, 12, 40, 32, 1.6, 40),
        # the single-material water phantom of the benchmark's configurations (no grid)
        _case("forward_water_128", "forward", (128, 128, 128), (1.0, 1.0, 1.0), 1, 60, 256, 256, 1.0, 61),
        # the headline configuration: a full rotation, two materials, a grid table per pixel
        _case("forward_grid_256", "forward", (256, 256, 256), (0.5, 0.5, 0.5), 2, 360, 512, 384, 0.8, 101,
              grid="pixel"),
        # the largest volume and detector of the configurations, four materials, part of a rotation
        _case("forward_4mat_512", "forward", (512, 512, 512), (0.4, 0.4, 0.4), 4, 48, 1024, 768, 0.4, 126,
              grid="column"),
        # the drop-in classes' default sampler (hardware texture), the reference's per-column grid table
        _case("forward_texture_256", "forward", (256, 256, 256), (0.5, 0.5, 0.5), 2, 90, 512, 384, 0.8, 101,
              mode="texture", grid="column"),
        # the same arithmetic in software on an odd-sized anisotropic volume, reversed rotation
        _case("forward_texemu_odd", "forward", (201, 187, 111), (0.6, 0.6, 0.9), 2, 75, 333, 217, 0.9, 81,
              mode="texemu", rot=-1),
        # a sparse phantom with empty-space skipping on
        _case("forward_skip_odd", "forward", (230, 230, 90), (0.5, 0.5, 0.8), 3, 45, 351, 175, 0.9, 71, skip=True),
        # host volumes in, host projections out
        _case("host_grid_256", "host", (256, 256, 256), (0.5, 0.5, 0.5), 2, 90, 512, 384, 0.8, 101, grid="pixel"),
        # one ordered-subset iteration: 12 of 360 views, forward and adjoint
        _case("subset_256", "subset", (256, 256, 256), (0.5, 0.5, 0.5), 1, 360, 512, 256, 0.8, 61, sub=12),
        # one algebraic step, small and ragged
        _case("lines_odd_97", "lines", (97, 113, 75), (0.8, 0.7, 1.1), 2, 41, 181, 117, 1.1, 0),
        # a training step through torch.autograd, three materials
        _case("train_3mat_256", "train", (256, 256, 256), (0.5, 0.5, 0.5), 3, 90, 384, 384, 1.0, 101, grid="pixel"),
        # uneven problems through one batched forward + loss + adjoint
        _case("batch_uneven_6", "batch", (64, 64, 64), (0.7, 0.7, 0.7), 3, 60, 128, 128, 0.9, 61, items=6, pick=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "forward", "host", "subset", "lines", "train", "fused", "batch"])
    mode = rng.choice(["trilinear", "trilinear", "trilinear", "texemu", "texture"])
    M = rng.choice([1, 2, 2, 3, 4])
    nx = _log(rng, 24, 400)
    ny = max(16, int(nx * rng.uniform(0.8, 1.2)))
    nz = max(12, int(nx * rng.uniform(0.3, 1.0)))
    vx = round(rng.uniform(0.3, 1.2), 3)
    vy = vx if rng.random() < 0.6 else round(vx * rng.uniform(0.8, 1.3), 3)
    vz = vx if rng.random() < 0.5 else round(vx * rng.uniform(0.8, 2.0), 3)
    U, V = _log(rng, 32, 900), _log(rng, 24, 600)
    sod = round(rng.uniform(900, 1100), 1)
    sdd = round(rng.uniform(1300, 1600), 1)
    pitch = round(rng.uniform(1.2, 1.7) * max(nx * vx, ny * vy) * sdd / sod / U, 4)
    views = _log(rng, 4, 360)
    c = _case("", kind, (nx, ny, nz), (vx, vy, vz), M, views, U, V, pitch, rng.randint(30, 126), mode=mode,
              grid=rng.choice(["none", "column", "pixel"]), det=rng.random() < 0.8,
              skip=kind == "forward" and rng.random() < 0.15, sub=0, items=rng.randint(2, 6) if kind == "batch" else 1,
              pick=rng.randint(0, 999), sod=sod, sdd=sdd, rot=rng.choice([1, 1, 1, -1]))
    if kind == "subset":
        c["sub"] = max(1, min(views, rng.randint(1, 16)))
    # no dearer than the largest listed case: fewer views, then fewer columns
    while _flops(c) > 3e11 and c["views"] > 4:
        c["views"] = max(4, c["views"] // 2)
        c["sub"] = min(c["sub"], c["views"])
    while _flops(c) > 3e11:
        c["U"], c["V"], c["pitch"] = c["U"] // 2, max(8, c["V"] // 2), c["pitch"] * 2
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# geometry, tables and phantoms

def _problems(case):
    """The case's problems: itself, or the batch's items (sizes around the case's own)."""
    if case["kind"] != "batch":
        return [dict(case)]
    r, out = random.Random(1000 + case["pick"]), []
    for k in range(case["items"]):
        c, f = dict(case), r.uniform(0.6, 2.0)
        c["nx"] = c["ny"] = max(16, int(case["nx"] * f))
        c["nz"] = max(12, int(case["nz"] * r.uniform(0.5, 1.6)))
        c["M"] = r.randint(1, min(3, max(1, case["M"])))
        c["views"] = max(3, int(case["views"] * r.uniform(0.4, 1.6)))
        c["U"], c["V"] = max(16, int(case["U"] * r.uniform(0.7, 2.0))), max(16, int(case["V"] * r.uniform(0.7, 1.8)))
        c["pitch"] = round(1.5 * c["nx"] * c["vx"] * c["sdd"] / c["sod"] / c["U"], 4)
        c["E"] = max(20, int(case["E"] * r.uniform(0.7, 1.5)))
        out.append(c)
    return out


def _geometry(c):
    return dict(pNumX=c["nx"], pNumY=c["ny"], pNumZ=c["nz"], pLengthX=c["nx"] * c["vx"], pLengthY=c["ny"] * c["vy"],
                pLengthZ=c["nz"] * c["vz"], projNum=c["views"], dNumU=c["U"], dNumV=c["V"], dSize=c["pitch"],
                sod=c["sod"], sdd=c["sdd"], rotatedDirection=c["rot"])


def _rng(seed, salt):
    return np.random.RandomState((int(seed) * 7919 + salt * 104729) % (1 << 31))


def _tables(c, seed, salt=0):
    """Spectrum [E], attenuation [E][M], grid and detector tables (FP32 host arrays)."""
    r = _rng(seed, salt)
    E = np.arange(20, 20 + c["E"], dtype=np.float64)
    top = E[-1] + 1
    S = np.clip(top - E, 0, None) / E * np.exp(-2.0 * (26500.0 * E ** -3 + 0.15) * 0.27)
    S = (S / S.sum()).astype(np.float32)
    amp = [4900.0, 30400.0, 95000.0, 2900.0]
    mu = np.stack([(amp[m] * r.uniform(0.95, 1.05) * E ** -3 + 0.16) / 10.0 for m in range(c["M"])], 1).astype(np.float32)
    U, V = c["U"], c["V"]
    G = D = None
    lay = {"none": 0, "column": 1, "pixel": 2}[c["grid"]]
    cov = torch.arange(c["E"], device=DEV, dtype=torch.float32).view(-1, 1, 1) / c["E"]
    u = torch.arange(U, device=DEV, dtype=torch.float32).view(1, 1, -1)
    v = torch.arange(V, device=DEV, dtype=torch.float32).view(1, -1, 1)
    ph = float(r.uniform(0, 6))
    if lay:
        G = 0.72 + 0.06 * cov + 0.02 * torch.sin(0.37 * u + ph)
        G = (G[:, 0] if lay == 1 else G - 0.03 * ((v - V / 2) / V) ** 2).contiguous().cpu().numpy()
    if c["det"]:
        D = ((0.9 - 0.55 * cov) * (1 + 0.03 * torch.sin(0.11 * u + 0.07 * v + ph))).contiguous().cpu().numpy()
    return S, mu, G, lay, D


def _volumes(c, seed, salt=0):
    """Density maps [nz][ny][nx], one per material: body, shells, inserts, rim."""
    r = _rng(seed, 31 + salt)
    x = ((torch.arange(c["nx"], device=DEV, dtype=torch.float32) + 0.5) / c["nx"] * 2 - 1).view(1, 1, -1)
    y = ((torch.arange(c["ny"], device=DEV, dtype=torch.float32) + 0.5) / c["ny"] * 2 - 1).view(1, -1, 1)
    z = ((torch.arange(c["nz"], device=DEV, dtype=torch.float32) + 0.5) / c["nz"] * 2 - 1).view(-1, 1, 1)
    rad = torch.sqrt((x / 0.88) ** 2 + (y / 0.68) ** 2)
    body = (rad <= 1) & (z.abs() <= 0.9)
    vols = [torch.zeros(c["nz"], c["ny"], c["nx"], device=DEV) for _ in range(c["M"])]
    vols[0][body] = 1.06
    for m in range(c["M"]):
        for _ in range(4):
            p, a = r.uniform(-0.5, 0.5, 3), r.uniform(0.08, 0.3, 3)
            q = ((x - p[0]) / a[0]) ** 2 + ((y - p[1]) / a[1]) ** 2 + ((z - p[2]) / a[2]) ** 2
            part = body & (q <= 1) & (q >= (0.4 if m == 1 else 0.0))
            vols[0][part] = float(r.uniform(0.2, 1.2)) if m == 0 else 0.0
            vols[m][part] = float(r.uniform(0.2, 1.9)) * (0.02 if m == 2 else 1.0)
    if c["M"] == 4:
        rim = body & (rad > 0.9)
        vols[0][rim] = 0.0
        vols[3][rim] = 0.92
    return vols


def _scalars(c):
    """The plan's derived geometry, FP32 in the reference's order of operations."""
    f = np.float32
    s = {k: f(v) for k, v in (("d", c["pitch"]), ("sod", c["sod"]), ("sdd", c["sdd"]), ("lx", c["nx"] * c["vx"]),
                              ("ly", c["ny"] * c["vy"]), ("lz", c["nz"] * c["vz"]))}
    s["hu"], s["hv"] = f(c["U"]) * s["d"] / f(2), f(c["V"]) * s["d"] / f(2)
    s["fov"] = s["sod"] * s["hu"] / np.sqrt(s["hu"] * s["hu"] + s["sdd"] * s["sdd"])
    s["px"], s["py"], s["pz"] = s["lx"] / f(c["nx"]), s["ly"] / f(c["ny"]), s["lz"] / f(c["nz"])
    s["dx"] = f(0.5 * float(s["px"]))
    s["K"] = int(np.floor(f(2) * s["fov"] / s["dx"] + f(0.5)))
    step = f(360) / f(c["views"])
    s["ang"] = [float(f(c["rot"]) * (f(p) * step / f(180) * f(math.acos(-1.0)))) for p in range(c["views"])]
    return s


def _rays(c, s, p):
    """FP64 voxel coordinates a + b i of every ray of view p, [V * U] per axis."""
    g = {k: float(s[k]) for k in ("d", "sod", "sdd", "hu", "hv", "fov", "dx", "px", "py", "pz", "lx", "ly", "lz")}
    du = (g["hu"] - g["d"] / 2 - torch.arange(c["U"], device=DEV, dtype=torch.float64) * g["d"]).view(1, -1)
    dv = (g["hv"] - g["d"] / 2 - torch.arange(c["V"], device=DEV, dtype=torch.float64) * g["d"]).view(-1, 1)
    R = torch.sqrt(g["sdd"] ** 2 + du * du + dv * dv)
    cg, cb = torch.sqrt(g["sdd"] ** 2 + du * du) / R, torch.sqrt(g["sdd"] ** 2 + dv * dv) / R
    A, B, C = cg * cb, cg * du / R, dv / R
    t0, dt, ct, st = g["sod"] - g["fov"] + g["dx"] / 2, g["dx"], math.cos(s["ang"][p]), math.sin(s["ang"][p])
    k = (A * ct - B * st, -(A * st + B * ct), -C)
    o = (-g["sod"] * ct + g["lx"] / 2, g["sod"] * st + g["ly"] / 2, g["lz"] / 2)
    return [((ki * t0 + oi) / g[pi]).expand(c["V"], c["U"]).reshape(-1) for ki, oi, pi in zip(k, o, ("px", "py", "pz"))], \
           [(ki * dt / g[pi]).expand(c["V"], c["U"]).reshape(-1) for ki, pi in zip(k, ("px", "py", "pz"))]


def _body_path(c, s, p):
    """Length (mm) of view p's rays inside a centred elliptical cylinder: the measured object."""
    a, b = _rays(c, s, p)
    n = (c["nx"], c["ny"])
    o = [(a[j] - n[j] / 2) / (0.41 * n[j]) for j in range(2)]
    d = [b[j] / (0.41 * n[j]) for j in range(2)]
    qa, qb, qc = d[0] ** 2 + d[1] ** 2, o[0] * d[0] + o[1] * d[1], o[0] ** 2 + o[1] ** 2 - 1
    return 2 * torch.sqrt(torch.clamp(qb * qb - qa * qc, min=0)) / qa * float(s["dx"])


def _weights64(tab):
    S, mu, G, lay, D = tab
    t = lambda x: torch.from_numpy(x).to(DEV).double()  # noqa: E731
    W = (I0VAL * t(S)).view(-1, 1, 1)
    if lay:
        W = W * (t(G)[:, None, :] if lay == 1 else t(G))
    return W * t(D) if D is not None else W


def _measured(c, tab, seed, views):
    """Measured intensities [views][V][U] of the elliptical object (FP32)."""
    s = _scalars(c)
    I0 = _weights64(tab).sum(0).expand(c["V"], c["U"])
    gen = torch.Generator(DEV).manual_seed(int(seed))
    path = torch.stack([_body_path(c, s, p).view(c["V"], c["U"]) for p in views])
    noise = torch.randn(path.shape, device=DEV, dtype=torch.float64, generator=gen)
    return (I0 * torch.exp(-0.018 * path + 0.02 * noise)).float().contiguous()


def _views(c):
    if c["kind"] != "subset":
        return range(c["views"])
    first = min(c["views"] // 3, c["views"] - c["sub"])
    return range(first, first + c["sub"])


# ---------------------------------------------------------------------------
# the timed passes

def _plan(c, tab):
    pr = Projector(_geometry(c), c["M"], c["mode"])
    if c["skip"]:
        pr.set_skip_empty(True)
    if tab is not None:
        S, mu, G, lay, D = tab
        pr.set_spectral_tables(S, mu, G, lay, D, I0VAL)
    return pr


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "plans": [], "vols": [], "target": []}
    for k, c in enumerate(_problems(case)):
        tab = None if kind == "lines" else _tables(c, seed, k)
        st["plans"].append(_plan(c, tab))
        st["vols"].append(_volumes(c, seed, k))
        if kind in ("subset", "train", "fused", "batch"):
            st["target"].append(_measured(c, tab, seed + k, _views(c)))
        if kind == "subset":
            st["range"] = (_views(c)[0], len(_views(c)))
        if kind == "lines":
            s = _scalars(c)
            path = torch.stack([_body_path(c, s, p).view(c["V"], c["U"]) for p in range(c["views"])])
            st["measured"] = (path[..., None] * torch.linspace(1.0, 0.2, c["M"], device=DEV, dtype=torch.float64)).float()
    if kind == "host":
        P, V, U = st["plans"][0].shape_proj
        st["host"] = [v.cpu().pin_memory() for v in st["vols"][0]]
        st["out"] = {"I": torch.empty((P, V, U)).pin_memory(), "IAbsorb": torch.empty((P, V, U)).pin_memory(),
                     "I0": torch.empty((V, U)).pin_memory()}
    if kind in ("train", "fused"):
        for v in st["vols"][0]:
            v.requires_grad_(True)
    if kind == "fused":
        st["loss"] = LogIntensityLoss(st["plans"][0])
    if kind == "batch":
        st["batch"] = Batch(st["plans"])
        st["grads"] = [[torch.zeros_like(v) for v in vs] for vs in st["vols"]]
        st["losses"] = torch.zeros(len(st["plans"]), device=DEV)
    torch.cuda.synchronize()
    return st


def run(st):
    kind, pr, vols = st["kind"], st["plans"][0], st["vols"][0]
    if kind == "forward":
        return pr.forward(vols)
    if kind == "host":
        return pr.forward_host(st["host"], out=st["out"])
    if kind == "subset":
        f = pr.forward(vols, want_L=True, views=st["range"])
        gI = f["I"] / st["target"][0] - 1.0
        return {"I": f["I"], "grads": pr.backward(f["L"], gI=gI, views=st["range"])}
    if kind == "lines":
        L = pr.line_integrals(vols)
        return {"L": L, "grads": pr.line_integrals_adjoint(L - st["measured"])}
    if kind == "batch":
        for gs in st["grads"]:
            for g in gs:
                g.zero_()
        r = st["batch"].forward_adjoint(st["vols"], st["target"], grads=st["grads"], loss=st["losses"])
        return {"grads": r["grads"], "loss": r["loss"]}
    for v in vols:
        v.grad = None
    if kind == "train":
        I, _, _ = project(pr, *vols)
        loss = torch.sum((torch.log(I) - torch.log(st["target"][0])) ** 2)
    else:
        loss = st["loss"](st["target"][0], *vols)
    loss.backward()
    return {"grads": [v.grad for v in vols], "loss": loss.detach()}


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _samples(c):
    """Ray samples inside the volume over the case's views (a subset of rays and views, scaled up)."""
    s = _scalars(c)
    views = list(_views(c))
    pick = views[::max(1, len(views) // 6)]
    u = (float(s["hu"]) - (np.linspace(0, c["U"] - 1, 33) + 0.5) * float(s["d"])).reshape(1, -1)
    v = (float(s["hv"]) - (np.linspace(0, c["V"] - 1, 17) + 0.5) * float(s["d"])).reshape(-1, 1)
    n = 0.0
    for p in pick:
        ct, st_ = math.cos(s["ang"][p]), math.sin(s["ang"][p])
        R = np.sqrt(c["sdd"] ** 2 + u * u + v * v)
        d = np.stack(np.broadcast_arrays((c["sdd"] * ct - u * st_) / R, -(c["sdd"] * st_ + u * ct) / R, -v / R), -1)
        o = np.array([-c["sod"] * ct, c["sod"] * st_, 0.0])
        half = np.array([c["nx"] * c["vx"], c["ny"] * c["vy"], c["nz"] * c["vz"]]) / 2
        with np.errstate(divide="ignore", invalid="ignore"):
            t1, t2 = (-half - o) / d, (half - o) / d
        near, far = np.minimum(t1, t2).max(-1), np.maximum(t1, t2).min(-1)
        n += float(np.maximum(far - near, 0).mean()) / float(s["dx"])
    return n / len(pick) * len(views) * c["U"] * c["V"]


def _flops(case):
    total = 0.0
    for c in _problems(case):
        n, rays = _samples(c), len(_views(c)) * c["U"] * c["V"]
        both = c["kind"] not in ("forward", "host")
        # trilinear: 8 multiply-adds per material and sample, again for the adjoint; the energy sum per ray
        total += n * c["M"] * 16 * (2 if both else 1) + (0 if c["kind"] == "lines" else rays * c["E"] * (2 * c["M"] + 6))
    return total


def work(case):
    nbytes = 0.0
    for c in _problems(case):
        vox, rays = c["nx"] * c["ny"] * c["nz"] * c["M"], len(_views(c)) * c["U"] * c["V"]
        both = c["kind"] not in ("forward", "host")
        nbytes += 4.0 * (vox * (2 if both else 1) + rays * (c["M"] * 2 if c["kind"] == "lines" else 2))
        nbytes += 4.0 * (0 if c["kind"] == "lines" else c["E"] * (c["U"] * c["V"] + c["M"]))
    return {"bytes": nbytes, "flops": _flops(case)}


# ---------------------------------------------------------------------------
# 64-bit restatement

class _March:
    """One problem's samples in FP64: footprint indices into a zero-padded volume and the 8 weights."""

    def __init__(self, c):
        self.c, self.s = c, _scalars(c)
        self.n = (c["nx"], c["ny"], c["nz"])
        self.dims = (c["nz"] + 4, c["ny"] + 4, c["nx"] + 4)
        self.off = [(dz * self.dims[1] + dy) * self.dims[2] + dx for dz in (0, 1) for dy in (0, 1) for dx in (0, 1)]

    def pad(self, vols):
        return [torch.nn.functional.pad(v.detach().double(), (2, 2, 2, 2, 2, 2)).reshape(-1) for v in vols]

    def unpad(self, flat):
        d = self.dims
        return flat.view(d)[2:d[0] - 2, 2:d[1] - 2, 2:d[2] - 2].contiguous()

    def _span(self, a, b):
        lo = torch.full_like(a[0], 0.0)
        hi = torch.full_like(a[0], float(self.s["K"]))
        for j in range(3):
            bj = torch.where(b[j].abs() < 1e-300, torch.full_like(b[j], 1e-300), b[j])
            t1, t2 = (-1.5 - a[j]) / bj, (self.n[j] + 0.5 - a[j]) / bj
            lo, hi = torch.maximum(lo, torch.minimum(t1, t2)), torch.minimum(hi, torch.maximum(t1, t2))
        live = hi >= lo
        if not bool(live.any()):
            return 0, 0
        return max(0, int(lo[live].min()) - 3), min(self.s["K"], int(hi[live].max()) + 4)

    def _coords32(self, p, i):
        """The FP32 sample coordinates of the texture modes (fused multiply-adds where they are defined as fused)."""
        c, s = self.c, self.s
        t = lambda x: torch.tensor(x, device=DEV, dtype=torch.float32)  # noqa: E731
        fma = lambda x, y, z: (x.double() * y.double() + z.double()).float()  # noqa: E731
        half, d = s["d"] / np.float32(2), t(s["d"])
        u = fma(-torch.arange(c["U"], device=DEV, dtype=torch.float32), d, t(s["hu"] - half)).view(1, -1)
        v = fma(-torch.arange(c["V"], device=DEV, dtype=torch.float32), d, t(s["hv"] - half)).view(-1, 1)
        s2, u2, v2 = t(s["sdd"] * s["sdd"]), u * u, v * v
        R = torch.sqrt((s2 + u2) + v2)
        sg, cg, sb, cb = v / R, torch.sqrt(s2 + u2) / R, u / R, torch.sqrt(s2 + v2) / R
        A, B, C = [x.expand(c["V"], c["U"]).reshape(1, -1) for x in (cg * cb, cg * sb, sg)]
        tt = fma(i.float().view(-1, 1), t(s["dx"]), t((s["sod"] - s["fov"]) + s["dx"] / np.float32(2)))
        ct, st = t(np.float32(math.cos(s["ang"][p]))), t(np.float32(math.sin(s["ang"][p])))
        X, Y, Z = fma(A, tt, t(-s["sod"])), B * tt, C * tt
        tu = fma(X, ct, -(Y * st)) + t(s["lx"] / np.float32(2))
        tv = -fma(X, st, Y * ct) + t(s["ly"] / np.float32(2))
        tw = -Z + t(s["lz"] / np.float32(2))
        return [q / t(s[k]) + 0.5 for q, k in ((tu, "px"), (tv, "py"), (tw, "pz"))]

    def steps(self, p, chunk):
        """(base index [k][rays], 8 weights) for blocks of samples of view p."""
        a, b = _rays(self.c, self.s, p)
        lo, hi = self._span(a, b)
        for i0 in range(lo, hi, chunk):
            i = torch.arange(i0, min(i0 + chunk, hi), device=DEV, dtype=torch.float64)
            if self.c["mode"] == "trilinear":
                base, fr = [], []
                for j in range(3):
                    x = torch.clamp(torch.addcmul(a[j], i.view(-1, 1), b[j]), -1.75, self.n[j] + 0.75)
                    f = torch.floor(x)
                    base.append(f)
                    fr.append(x - f)
                w = [(1 - fr[0], fr[0]), (1 - fr[1], fr[1]), (1 - fr[2], fr[2])]
                yz = [w[2][dz] * w[1][dy] for dz in (0, 1) for dy in (0, 1)]
                ws = [yz[k >> 1] * w[0][k & 1] for k in range(8)]
            else:
                q = [torch.floor(x.double() * 256.0 - 127.5) for x in self._coords32(p, i)]
                q = [torch.clamp(x, -448.0, self.n[j] * 256.0 + 191.0) for j, x in enumerate(q)]
                base = [torch.floor(x / 256) for x in q]
                fa, fb, fc = [x - 256 * f for x, f in zip(q, base)]
                ws = []
                for z in (256 - fc, fc):
                    p1 = torch.floor((fa * z + 128) / 256)
                    p0 = z - p1
                    w11, w01 = torch.floor((fb * p1 + 128) / 256), torch.floor((fb * p0 + 127) / 256)
                    ws += [(p0 - w01) / 256, (p1 - w11) / 256, w01 / 256, w11 / 256]
            idx = ((base[2] + 2) * self.dims[1] + (base[1] + 2)) * self.dims[2] + (base[0] + 2)
            yield idx.long(), ws

    def lines(self, pads, p):
        L = torch.zeros(self.c["V"] * self.c["U"], len(pads), device=DEV, dtype=torch.float64)
        for idx, ws in self.steps(p, self._chunk()):
            for k in range(8):
                at = idx + self.off[k]
                for m, v in enumerate(pads):
                    L[:, m] += (ws[k] * v[at]).sum(0)
        return L * float(self.s["dx"])

    def scatter(self, gL, grads, p):
        gL = gL * float(self.s["dx"])
        for idx, ws in self.steps(p, self._chunk()):
            for k in range(8):
                at = (idx + self.off[k]).reshape(-1)
                for m, g in enumerate(grads):
                    g.index_add_(0, at, (ws[k] * gL[:, m]).reshape(-1))

    def _chunk(self):
        return max(1, 4_000_000 // (self.c["U"] * self.c["V"]))


def exact(case, seed):
    total = 0.0
    probs = _problems(case)
    for c in probs:
        total += _samples(c) * (1 + 0.6 * c["M"]) * (1 if c["kind"] in ("forward", "host") else 3)
    if total > 1.4e10:
        return None
    res = []
    for k, c in enumerate(probs):
        kind, views = c["kind"], list(_views(c))
        m = _March(c)
        pads = m.pad(_volumes(c, seed, k))
        both = kind not in ("forward", "host")
        grads = [torch.zeros_like(v) for v in pads] if both else []
        V, U = c["V"], c["U"]
        if kind == "lines":
            Ls = []
            for p in views:
                L = m.lines(pads, p)
                Ls.append(L.view(V, U, -1))
                meas = (_body_path(c, m.s, p)[:, None] * torch.linspace(1.0, 0.2, c["M"], device=DEV, dtype=torch.float64)).float()
                m.scatter(L - meas.double(), grads, p)
            return {"L": torch.stack(Ls), "grads": [m.unpad(g) for g in grads]}
        tab = _tables(c, seed, k)
        W = _weights64(tab).expand(c["E"], V, U).reshape(c["E"], -1)
        mu = torch.from_numpy(tab[1]).to(DEV).double()
        T = _measured(c, tab, seed + k, views).double().view(len(views), -1) if both else None
        Is, As = [], []
        for j, p in enumerate(views):
            L = m.lines(pads, p)
            I, A = torch.zeros(V * U, device=DEV, dtype=torch.float64), torch.zeros(V * U, device=DEV, dtype=torch.float64)
            S = torch.zeros_like(L)
            for e in range(c["E"]):
                att = L @ mu[e]
                w = W[e] * torch.exp(-att)
                I += w
                A -= W[e] * torch.expm1(-att)
                if both:
                    S += w[:, None] * mu[e]
            Is.append(I.view(V, U))
            As.append(A.view(V, U))
            if both:
                gI = I / T[j] - 1 if kind == "subset" else 2 * (torch.log(I) - torch.log(T[j])) / I
                m.scatter(-gI[:, None] * S, grads, p)
        g = [m.unpad(x) for x in grads]
        if not both:
            return {"I": torch.stack(Is), "IAbsorb": torch.stack(As), "I0": W.sum(0).view(V, U)}
        if kind == "subset":
            return {"I": torch.stack(Is), "grads": g}
        if kind in ("train", "fused"):
            return {"grads": g, "loss": None}  # the loss is summed in no fixed order
        res.append(g)
    return {"grads": res, "loss": None}
