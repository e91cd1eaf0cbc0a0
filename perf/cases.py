"""Workloads of the interpolation library, called through its public entry points.

Each case is one call pattern of a program that uses partia_b200, at the sizes
of the repository's configurations (uniform box, Plummer sphere, clumps, disc
with halo) or around them:

  kind "points"   Context.interp_points on device arrays
  kind "api"      PointSamples_interpolation on host arrays (the Partia interface)
  kind "grid"     Context.interp_grid, and with "box" an oriented box beside it
  kind "lines"    Context.interp_lines on device arrays
  kind "beam"     Context.interp_beam (column density of a parallel beam)
  kind "density"  set_particles + build + density: one round of the h iteration
  kind "adjoint"  Context.adjoint_grid / adjoint_points
  kind "train"    autograd.interpolate_beam forward and backward (one step of a
                  fit: new particle values on every step)

Particles come from the seed alone; h and rho from the model's own density
(h = 1.2 (m / rho)^(1/3)), so every sample near the model has the 50 to 100
neighbours that the method is used with.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "partia.jl_b200"))

import partia_b200 as P  # noqa: E402
from partia_b200 import _lib as L  # noqa: E402
from partia_b200 import autograd as AG  # noqa: E402

F64 = torch.float64
KERNELS = {"M4": P.M4_spline, "M5": P.M5_spline, "M6": P.M6_spline, "C2": P.C2_Wendland, "C4": P.C4_Wendland,
           "C6": P.C6_Wendland}
SUPPORT = {"M4": 2.0, "M5": 2.5, "M6": 3.0, "C2": 2.0, "C4": 2.0, "C6": 2.0}
NORM3 = {"M4": 1 / math.pi, "M5": 0.05 / math.pi, "M6": 1 / (120 * math.pi), "C2": 21 / (16 * math.pi),
         "C4": 495 / (256 * math.pi), "C6": 1365 / (512 * math.pi)}
STRATEGY = {"gather": L.PSB_GATHER, "scatter": L.PSB_SCATTER, "symmetric": L.PSB_SYMMETRIC}
# the output sets: rho and a Shepard mean; rho, grad rho, div A, curl A (8
# fields); the same with a Shepard scalar of its own
CATALOGS = {
    "rho": dict(scalars=[0], shepard=[0]),
    "scalars": dict(scalars=[0, 1], shepard=[0, 1]),
    "mean": dict(scalars=[1], shepard=[1]),
    "full": dict(scalars=[0], shepard=[0], grads=[0], divs=[1, 2, 3], curls=[1, 2, 3]),
    "disc": dict(scalars=[0, 4], shepard=[0, 1], grads=[0], curls=[1, 2, 3]),
}


def listed():
    return [
        # a few probe points in a small set: what one call costs (latency, launches)
        dict(name="probe_points", kind="points", model="plummer", n=60_000, ns=37, kernel="M5", cat="full",
             strategy="symmetric", fp32c=False),
        # the Partia interface on host arrays, with its default kernel and precision
        dict(name="api_points", kind="api", model="clumps", n=150_000, ns=50_001, kernel="M5", cat="scalars",
             strategy="symmetric", fp32c=False),
        # the uniform-box configuration: gather, rho and a Shepard mean on cell centres
        dict(name="grid_uniform_gather", kind="grid", model="uniform", n=100_000, nx=64, ny=64, nz=64, box=0,
             kernel="M4", cat="scalars", strategy="gather", fp32c=False),
        # an ordinary ragged grid in double precision, all derivative fields
        dict(name="grid_ragged_fp64", kind="grid", model="plummer", n=500_000, nx=101, ny=67, nz=53, box=0,
             kernel="M4", cat="full", strategy="symmetric", fp32c=False),
        # the Plummer configuration: 2M particles, 8 fields on 128^3
        dict(name="grid_plummer_fp32c", kind="grid", model="plummer", n=2_000_000, nx=128, ny=128, nz=128, box=0,
             kernel="M4", cat="full", strategy="symmetric", fp32c=True),
        # unordered samples on the device (tracers), a smoother kernel
        dict(name="points_tracers_fp32c", kind="points", model="plummer", n=1_000_000, ns=700_003, kernel="C4",
             cat="full", strategy="symmetric", fp32c=True),
        # float32 particle data: a grid and an oriented box, as in the disc + halo configuration
        dict(name="grid_box_float32", kind="grid", model="disc", n=4_000_000, nx=128, ny=128, nz=128, box=64,
             kernel="M4", cat="disc", strategy="symmetric", fp32c=True),
        # the column-density image of the clump configuration
        dict(name="beam_clumps_fp32c", kind="beam", model="clumps", n=8_000_000, nx=1024, ny=1024, kernel="M4",
             cat="rho", strategy="scatter", fp32c=True),
        # arbitrary sight lines in double precision
        dict(name="lines_sightlines_fp64", kind="lines", model="clumps", n=300_000, ns=20_011, kernel="M5",
             cat="scalars", strategy="scatter", fp32c=False),
        # one round of the smoothing-length iteration: upload, tree, density at the particles
        dict(name="density_round", kind="density", model="clumps", n=1_000_000, kernel="M4", strategy="gather",
             fp32c=False),
        # gradients of a loss on every field of the Plummer configuration
        dict(name="adjoint_grid_full", kind="adjoint", model="plummer", n=2_000_000, nx=128, ny=128, nz=128,
             kernel="M4", cat="full", strategy="symmetric"),
        # a fit to a column-density map: forward, loss, gradients, new particles each step
        dict(name="train_beam", kind="train", model="clumps", n=1_000_000, nx=512, ny=512, kernel="M4", cat="rho"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["points", "api", "grid", "grid", "lines", "beam", "density", "adjoint", "train"])
    c = dict(kind=kind, model=rng.choice(["plummer", "uniform", "clumps"]),
             kernel=rng.choice(["M4", "M4", "M5", "M6", "C2", "C4", "C6"]))
    if kind == "points":
        c.update(n=size(2_000, 1_500_000), ns=size(1, 700_000), cat=rng.choice(["scalars", "full"]),
                 strategy=rng.choice(list(STRATEGY)), fp32c=rng.random() < 0.5)
    elif kind == "api":
        c.update(n=size(2_000, 200_000), ns=size(8, 80_000), cat=rng.choice(["scalars", "full"]),
                 strategy=rng.choice(list(STRATEGY)), fp32c=rng.random() < 0.3)
    elif kind == "grid":
        c.update(n=size(5_000, 2_000_000), nx=size(9, 110), ny=size(9, 110), nz=size(5, 110), box=0,
                 cat=rng.choice(["rho", "scalars", "full"]), strategy=rng.choice(list(STRATEGY)),
                 fp32c=rng.random() < 0.5)
        if rng.random() < 0.3:
            c.update(model="disc", kernel="M4", cat="disc", box=rng.choice([0, 24, 48]))
    elif kind == "lines":
        c.update(n=size(3_000, 150_000), ns=size(10, 12_000), cat=rng.choice(["rho", "scalars"]), strategy="scatter",
                 fp32c=rng.random() < 0.5)
    elif kind == "beam":
        c.update(n=size(5_000, 3_000_000), nx=size(33, 700), ny=size(33, 700), cat=rng.choice(["rho", "scalars"]),
                 strategy="scatter", fp32c=rng.random() < 0.6, kernel=rng.choice(["M4", "M4", "C2"]))
    elif kind == "density":
        c.update(n=size(3_000, 1_500_000), strategy=rng.choice(["gather", "gather", "symmetric"]),
                 fp32c=rng.random() < 0.3)
    elif kind == "adjoint":
        c.update(n=size(3_000, 700_000), nx=size(5, 70), ny=size(5, 70), nz=size(5, 70),
                 cat=rng.choice(["mean", "scalars", "full"]), strategy=rng.choice(list(STRATEGY)))
        if rng.random() < 0.4:  # explicit points instead of a grid
            c.update(ns=size(50, 200_000))
    else:
        c.update(n=size(5_000, 700_000), nx=size(33, 400), ny=size(33, 400), cat=rng.choice(["rho", "scalars"]),
                 kernel=rng.choice(["M4", "M4", "C2"]))
    return c


# ---------------------------------------------------------------------------
# particle models
# ---------------------------------------------------------------------------
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1_000_003 + salt) % (1 << 62))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=F64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=F64)


def _isotropic(g, r):
    n = r.numel()
    cz = 2 * _rand(g, n) - 1
    phi = 2 * math.pi * _rand(g, n)
    s = torch.sqrt(1 - cz * cz)
    return r * s * torch.cos(phi), r * s * torch.sin(phi), r * cz


def _plummer(g, n, a):
    """Plummer positions, truncated at 10 a (mass fraction (1 + 1/100)^(-3/2))."""
    u = _rand(g, n).clamp_min(1e-12) * (1 + 0.01) ** -1.5
    return _isotropic(g, a / torch.sqrt(u ** (-2.0 / 3.0) - 1))


def _clump_model(seed):
    g = _gen(seed, 77)
    w = -torch.log(_rand(g, 64).clamp_min(1e-12))
    sig = torch.exp(math.log(0.005) + (math.log(0.05) - math.log(0.005)) * _rand(g, 64))
    return w / w.sum(), _rand(g, 64, 3), sig


def _positions(model, n, g, seed):
    if model == "uniform":
        return [_rand(g, n) for _ in range(3)]
    if model == "plummer":
        return list(_plummer(g, n, 0.1))
    if model == "clumps":
        w, cen, sig = _clump_model(seed)
        nc = int(round(0.9 * n))
        lab = torch.searchsorted(torch.cumsum(w, 0), _rand(g, nc)).clamp_max(63)
        p = torch.cat([cen[lab] + sig[lab, None] * _randn(g, nc, 3), _rand(g, n - nc, 3)])
        return [p[:, k].contiguous() for k in range(3)]
    nd = int(round(0.7 * n))  # disc + halo
    R = -0.2 * torch.log((_rand(g, nd) * _rand(g, nd)).clamp_min(1e-12))
    phi = 2 * math.pi * _rand(g, nd)
    z = 0.02 * torch.atanh((2 * _rand(g, nd) - 1).clamp(-1 + 1e-9, 1 - 1e-9))
    hx, hy, hz = _plummer(g, n - nd, 0.3)
    return [torch.cat([R * torch.cos(phi), hx]), torch.cat([R * torch.sin(phi), hy]), torch.cat([z, hz])]


def _density(model, x, y, z, seed):
    """The model's density at unit total mass."""
    if model == "uniform":
        return torch.ones_like(x)

    def plummer(a):
        return 3 / (4 * math.pi * a ** 3) * (1 + (x * x + y * y + z * z) / a ** 2) ** -2.5 * 1.01 ** 1.5

    if model == "plummer":
        return plummer(0.1)
    if model == "clumps":
        w, cen, sig = _clump_model(seed)
        rho = torch.full_like(x, 0.1)
        for k in range(64):
            d2 = (x - cen[k, 0]) ** 2 + (y - cen[k, 1]) ** 2 + (z - cen[k, 2]) ** 2
            rho += 0.9 * w[k] / (2 * math.pi * sig[k] ** 2) ** 1.5 * torch.exp(-0.5 * d2 / sig[k] ** 2)
        return rho
    R = torch.sqrt(x * x + y * y)
    disc = torch.exp(-R / 0.2) / (2 * math.pi * 0.04) / (2 * 0.02) / torch.cosh((z / 0.02).clamp(-300, 300)) ** 2
    return 0.7 * disc + 0.3 * plummer(0.3)


def _particles(c, seed):
    """x y z m h rho and the columns (rho, a vector field, a scalar)."""
    g = _gen(seed, 1)
    n, model = c["n"], c["model"]
    x, y, z = _positions(model, n, g, seed)
    rho = _density(model, x, y, z, seed)
    m = torch.full_like(x, 1.0 / n)
    h = 1.2 * (m / rho) ** (1.0 / 3.0) * (1 + 0.05 * (2 * _rand(g, n) - 1))
    rho = rho * (1 + 0.02 * _randn(g, n)).clamp(0.9, 1.1)
    ax, ay, az = -y + 0.01 * _randn(g, n), x + 0.01 * _randn(g, n), 0.1 * z + 0.01 * _randn(g, n)
    if c["kind"] in ("points", "grid", "adjoint", "api") and c["cat"] in ("full", "disc"):
        cols = [rho.clone(), ax, ay, az] + ([z * z] if c["cat"] == "disc" else [])
    else:
        cols = [rho.clone(), torch.sin(6 * x) * torch.cos(6 * y) + z]
        if c.get("cat") == "rho":
            cols = cols[:1]
    if model == "disc":  # float32 particle data
        x, y, z, m, h, rho = (t.float() for t in (x, y, z, m, h, rho))
        cols = [t.float() for t in cols]
    return dict(x=x, y=y, z=z, m=m, h=h, rho=rho, cols=cols)


def _scatter_points(c, ns, seed):
    """Sample positions that follow the model (tracers): a displaced draw of it."""
    g = _gen(seed, 2)
    p = _positions(c["model"], ns, g, seed)
    return [(t + 0.01 * _randn(g, ns)).contiguous() for t in p]


def _cat(c):
    return P.CatalogC(**CATALOGS[c["cat"]])


def _axes(c, dtype=np.float64):
    lo, hi = (0.0, 1.0) if c["model"] in ("uniform", "clumps") else (-0.5, 0.5)
    out = []
    for n in (c["nx"], c["ny"], c["nz"]):
        d = (hi - lo) / n
        out.append(P.linrange(lo + 0.5 * d, hi - 0.5 * d, n, dtype))
    return out


def _box(seed):
    """Frame of an oriented box around the disc's centre (position, right, up, forward) and its extents."""
    a = 0.3 + 0.01 * (seed % 50)
    ca, sa = math.cos(a), math.sin(a)
    fr = np.array([0.0, 0.0, 0.0, ca, sa, 0.0, -sa * 0.8, ca * 0.8, 0.6, sa * 0.6, -ca * 0.6, 0.8])
    return fr.astype(np.float32), np.array([-0.3, 0.3, -0.25, 0.25, -0.1, 0.1], dtype=np.float32)


def _beam():
    """The beam's frame: 30 degrees about z, then 45 degrees about x; it covers the unit box's middle."""
    c30, s30, c45 = math.cos(math.pi / 6), math.sin(math.pi / 6), math.sqrt(0.5)
    r = np.array([c30, s30, 0.0])
    u = np.array([-s30 * c45, c30 * c45, c45])
    f = np.cross(r, u)
    return np.concatenate([[0.5, 0.5, 0.5], r, u, f])


def _beam_params(c):
    w = 0.5 if c["model"] in ("uniform", "clumps") else 0.4
    return np.array([-w, w, -w, w])


def _beam_frame(c):
    fr = _beam()
    if c["model"] not in ("uniform", "clumps"):
        fr[:3] = 0.0
    return fr


def _sight_lines(c, seed):
    """Lines through the model in random directions (origins near a random particle's place)."""
    g = _gen(seed, 3)
    o = _positions(c["model"], c["ns"], g, seed)
    o = [t + 0.02 * _randn(g, c["ns"]) for t in o]
    d = _randn(g, 3, c["ns"])
    d = d / torch.sqrt((d * d).sum(0))
    return o, [d[k].contiguous() for k in range(3)]


def _prec(c):
    return L.PSB_PREC_FP32C if c["fp32c"] else L.PSB_PREC_FP64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    p = _particles(c, seed)
    s = dict(c=c, p=p)
    if kind == "api":
        host = {k: (p[k].cpu().numpy() if k != "cols" else [t.cpu().numpy() for t in p[k]]) for k in p}
        if c["cat"] == "full":
            names, q = ("rho", "Ax", "Ay", "Az"), dict(scalars=("rho",), gradients=("rho",), divergences=("A",),
                                                       curls=("A",))
        else:
            names, q = ("rho", "T"), dict(scalars=("rho", "T"))
        s["backend"] = P.B200ComputeBackend(0, _prec(c))
        s["input"], s["catalog"] = P.build_input(
            s["backend"], *(host[k] for k in ("x", "y", "z", "m", "h", "rho")), host["cols"], column_names=names,
            smoothed_kernel=KERNELS[c["kernel"]], **q)
        s["lbvh"] = P.LinearBVH_(s["input"], s["backend"])
        s["strategy"] = dict(gather=P.itpGather, scatter=P.itpScatter, symmetric=P.itpSymmetric)[c["strategy"]]
        coor = tuple(t.cpu().numpy() for t in _scatter_points(c, c["ns"], seed))
        s["samples"] = P.PointSamples(np.zeros(c["ns"]), coor)
        torch.cuda.synchronize()
        return s
    if kind == "train":
        s["leaf"] = {k: p[k].clone().requires_grad_(True) for k in ("x", "y", "z", "m")}
        s["cols"] = [t.clone().requires_grad_(True) for t in p["cols"]]
        g = _gen(seed, 4)
        nout = _cat(c).L
        s["target"] = _rand(g, nout, c["nx"] * c["ny"])
        torch.cuda.synchronize()
        return s
    s["ctx"] = P.Context(0)
    if kind != "density":
        s["cat"] = _cat(c)
        torch.cuda.synchronize()
        _load(s)
    if kind == "points":
        s["samples"] = _scatter_points(c, c["ns"], seed)
    elif kind == "grid":
        s["axes"] = _axes(c, np.float32 if c["model"] == "disc" else np.float64)
        s["box"] = _box(seed)
    elif kind == "lines":
        s["lines"] = _sight_lines(c, seed)
    elif kind == "adjoint":
        if "ns" in c:
            s["samples"] = _scatter_points(c, c["ns"], seed)
            ns = c["ns"]
        else:
            s["axes"] = _axes(c)
            ns = c["nx"] * c["ny"] * c["nz"]
        g = _gen(seed, 4)
        s["gout"] = [_randn(g, ns) for _ in range(s["cat"].L)]
    torch.cuda.synchronize()
    return s


def _load(s):
    p, ctx = s["p"], s["ctx"]
    ctx.set_particles(p["x"], p["y"], p["z"], p["m"], p["h"], p["rho"], p["cols"],
                      kernel=KERNELS[s["c"]["kernel"]].code)
    ctx.build(want_perm=False)


def run(state):
    s = state
    c, kind = s["c"], s["c"]["kind"]
    if kind == "points":
        return s["ctx"].interp_points(*s["samples"], s["cat"], strategy=STRATEGY[c["strategy"]], prec=_prec(c))
    if kind == "api":
        out = P.PointSamples_interpolation(s["backend"], s["samples"], s["input"], s["lbvh"], s["catalog"],
                                           s["strategy"])
        return [g.grid for g in out.grids]
    if kind == "grid":
        st = STRATEGY[c["strategy"]]
        out = s["ctx"].interp_grid(*s["axes"], s["cat"], strategy=st, prec=_prec(c), device_out=True)
        if c["box"]:
            b = c["box"]
            out = out + s["ctx"].interp_box(*s["box"], b, b, b, s["cat"], strategy=st, prec=_prec(c), device_out=True)
        return out
    if kind == "lines":
        return s["ctx"].interp_lines(*s["lines"], s["cat"], prec=_prec(c))
    if kind == "beam":
        return s["ctx"].interp_beam(_beam_frame(c), _beam_params(c), c["nx"], c["ny"], s["cat"], prec=_prec(c),
                                    device_out=True)
    if kind == "density":
        p, ctx = s["p"], s["ctx"]
        ctx.set_particles(p["x"], p["y"], p["z"], p["m"], p["h"], p["rho"], kernel=KERNELS[c["kernel"]].code)
        ctx.build(want_perm=False)
        return ctx.density(p["x"], p["y"], p["z"], strategy=STRATEGY[c["strategy"]], hmode=L.PSB_H_PER_SAMPLE,
                           hs=p["h"], prec=_prec(c))
    if kind == "adjoint":
        st = STRATEGY[c["strategy"]]
        if "ns" in c:
            return s["ctx"].adjoint_points(*s["samples"], s["cat"], s["gout"], strategy=st)
        return s["ctx"].adjoint_grid(*s["axes"], s["cat"], s["gout"], strategy=st, device=True)
    leaf, cols, p = s["leaf"], s["cols"], s["p"]
    out = AG.interpolate_beam(leaf["x"], leaf["y"], leaf["z"], leaf["m"], p["h"], p["rho"], cols, _beam_frame(c),
                              _beam_params(c), c["nx"], c["ny"], _cat(c), kernel=KERNELS[c["kernel"]].code)
    r = torch.nan_to_num(out) - s["target"]
    loss = 0.5 * (r * r).sum()
    grads = torch.autograd.grad(loss, [leaf["m"], leaf["x"], leaf["y"], leaf["z"], *cols])
    return [out.detach(), loss.detach(), *grads]


def work(case):
    """Bytes: particles and samples read once, outputs written once.  Operations:
    the pairs inside the supports at h = 1.2 (m / rho)^(1/3) (a line of a
    clump model crosses about 7 N^(1/3) supports), times the arithmetic of one pair."""
    c = case
    kind, n = c["kind"], c["n"]
    w = 4 if c["model"] == "disc" else 8
    spec = CATALOGS[c.get("cat", "rho")]
    kc = {"rho": 1, "scalars": 2, "mean": 1, "full": 4, "disc": 5}[c.get("cat", "rho")]
    grads = "grads" in spec or "divs" in spec
    nout = len(spec["scalars"]) + 3 * len(spec.get("grads", ())) + (1 if "divs" in spec else 0) + \
        (3 if "curls" in spec else 0)
    line = kind in ("lines", "beam", "train")
    if "ns" in c:
        ns = c["ns"]
    elif kind == "density":
        ns = n
    elif line:
        ns = c["nx"] * c["ny"]
    else:
        ns = c["nx"] * c["ny"] * c["nz"] + c.get("box", 0) ** 3
    nin = 0 if kind in ("grid", "beam", "train") else (6 if kind == "lines" else 3)
    bytes_ = w * (n * (6 + (0 if kind == "density" else kc)) + ns * (nin + (1 if kind == "density" else nout)))
    K = SUPPORT[c["kernel"]]
    pairs = ns * (7.0 * n ** (1 / 3) * (K / 2) ** 2 if line else 4.19 * (1.2 * K) ** 3)
    if kind == "density":
        per = 25
    elif grads:
        per = 45 + 8 * kc
    else:
        per = 25 + 2 * kc
    flops = pairs * per
    if kind in ("adjoint", "train"):  # the gradients: both ways of every pair, one output per particle and input
        flops *= 3
        bytes_ += w * (n * (4 + kc) + ns * nout)
    return {"bytes": float(bytes_), "flops": float(flops)}


# ---------------------------------------------------------------------------
# 64-bit values by direct sums over the pairs
# ---------------------------------------------------------------------------
def _kernel(k, q):
    """f(q) and f'(q) of the dimensionless kernel."""
    if k in ("C2", "C4", "C6"):
        a = (1 - 0.5 * q).clamp_min(0)
        if k == "C2":
            return a ** 4 * (2 * q + 1), -5 * q * a ** 3
        if k == "C4":
            return a ** 6 * (35 / 12 * q * q + 3 * q + 1), -14 / 3 * q * (1 + 2.5 * q) * a ** 5
        return (a ** 8 * (4 * q ** 3 + 6.25 * q * q + 4 * q + 1), -5.5 * q * (1 + 3.5 * q + 4 * q * q) * a ** 7)
    pw, co, e = {"M4": (3, (0.25, -1.0), (2.0, 1.0)), "M5": (4, (1.0, -5.0, 10.0), (2.5, 1.5, 0.5)),
                 "M6": (5, (1.0, -6.0, 15.0), (3.0, 2.0, 1.0))}[k]
    f = sum(a * (b - q).clamp_min(0) ** pw for a, b in zip(co, e))
    return f, sum(-pw * a * (b - q).clamp_min(0) ** (pw - 1) for a, b in zip(co, e))


def _groups(s, size):
    """Groups of nearby samples (indices), by a coarse Morton key."""
    lo = torch.stack([t.min() for t in s])
    ext = torch.stack([t.max() for t in s]) - lo
    key = torch.zeros(s[0].numel(), dtype=torch.int64, device="cuda")
    for d in range(3):
        q = ((s[d] - lo[d]) / ext[d].clamp_min(1e-300) * 1023).long().clamp(0, 1023)
        for b in range(10):
            key |= ((q >> b) & 1) << (3 * b + d)
    return torch.split(torch.argsort(key, stable=True), size)


def _near(x, lo, hi, r):
    d2 = sum(torch.clamp(torch.maximum(lo[d] - x[d], x[d] - hi[d]), min=0) ** 2 for d in range(3))
    return torch.nonzero(d2 <= r * r)[:, 0]


def _nearest_h(s, x, h):
    ha = torch.empty_like(s[0])
    for g in _groups(s, 1024):
        sg = [t[g] for t in s]
        lo, hi = torch.stack([t.min() for t in sg]), torch.stack([t.max() for t in sg])
        cen, rad = 0.5 * (lo + hi), 0.5 * torch.sqrt(((hi - lo) ** 2).sum())
        d = torch.sqrt(sum((x[k] - cen[k]) ** 2 for k in range(3)))
        cand = torch.nonzero(d <= (2 * rad + d.min()) * (1 + 1e-12))[:, 0]
        best = torch.full_like(sg[0], math.inf)
        for cc in torch.split(cand, 1 << 17):
            d2 = sum((sg[k][:, None] - x[k][cc][None, :]) ** 2 for k in range(3))
            v, i = d2.min(1)
            ha[g] = torch.where(v < best, h[cc][i], ha[g])
            best = torch.minimum(v, best)
    return ha


def _pairs(s, ha, x, h, K, strategy, size=1024):
    """(sample, particle) indices of the pairs, group by group."""
    for g in _groups(s, size):
        sg = [t[g] for t in s]
        lo, hi = torch.stack([t.min() for t in sg]), torch.stack([t.max() for t in sg])
        r = {"gather": K * ha[g].max() if ha is not None else None, "scatter": K * h}.get(strategy)
        if strategy == "symmetric":
            r = K * torch.maximum(h, ha[g].max())
        cand = _near(x, lo, hi, r)
        for cc in torch.split(cand, 1 << 16):
            d2 = sum((sg[k][:, None] - x[k][cc][None, :]) ** 2 for k in range(3))
            ra = K * (ha[g][:, None] if strategy == "gather" else
                      h[cc][None, :] if strategy == "scatter" else torch.maximum(ha[g][:, None], h[cc][None, :]))
            i, j = torch.nonzero(d2 <= ra * ra, as_tuple=True)
            if i.numel():
                yield g[i], cc[j]


def _weights(kernel, d, ha, hb, strategy):
    """W and grad W / d of pairs with separations d."""
    r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
    rs = torch.where(r > 0, r, torch.ones_like(r))
    sg = NORM3[kernel]

    def one(h):
        f, df = _kernel(kernel, r / h)
        return sg * f / h ** 3, sg * df / h ** 4 / rs
    if strategy == "gather":
        return one(ha)
    if strategy == "scatter":
        return one(hb)
    (a, b), (e, f) = one(ha), one(hb)
    return 0.5 * (a + e), 0.5 * (b + f)


def _fields(c, s, x, m, h, rho, cols, spec):
    """The catalog's fields at samples s, in catalog order."""
    K, st, ns = SUPPORT[c["kernel"]], c["strategy"], s[0].numel()
    ha = _nearest_h(s, x, h) if st != "scatter" else None
    mr = m / rho
    zero = lambda *k: torch.zeros(*k, ns, dtype=F64, device="cuda")  # noqa: E731
    S1, G, Sw, Sg = zero(), zero(3), zero(len(cols)), zero(len(cols), 3)
    for i, j in _pairs(s, ha, x, h, K, st):
        d = [s[k][i] - x[k][j] for k in range(3)]
        W, gw = _weights(c["kernel"], d, None if ha is None else ha[i], h[j], st)
        w, g = mr[j] * W, mr[j] * gw
        S1.index_add_(0, i, w)
        for k in range(3):
            G[k].index_add_(0, i, g * d[k])
        for q, A in enumerate(cols):
            Sw[q].index_add_(0, i, A[j] * w)
            if "grads" in spec:
                for k in range(3):
                    Sg[q, k].index_add_(0, i, A[j] * g * d[k])
    empty = S1 == 0
    S1 = torch.where(empty, torch.full_like(S1, math.nan), S1)
    out = [Sw[q] / S1 if n else Sw[q] + 0 * S1 for q, n in zip(spec["scalars"], spec["shepard"])]
    D = lambda q, k: Sg[q, k] - G[k] * Sw[q] / S1  # noqa: E731  the derivative of column q along k
    for q in spec.get("grads", ()):
        out += [D(q, k) for k in range(3)]
    if "divs" in spec:
        out.append(sum(D(q, k) for k, q in enumerate(spec["divs"])))
    if "curls" in spec:
        a, b, e = spec["curls"]
        out += [D(e, 1) - D(b, 2), D(a, 2) - D(e, 0), D(b, 0) - D(a, 1)]
    return out


def _line_table(kernel, n=4096):
    """The line integral of the kernel at n points of [0, K], by Gauss-Legendre on each smooth piece."""
    K = SUPPORT[kernel]
    brk = {"M4": (1, 2), "M5": (0.5, 1.5, 2.5), "M6": (1, 2, 3)}.get(kernel, (2,))
    gx, gw = (torch.from_numpy(v).cuda() for v in np.polynomial.legendre.leggauss(64))
    b = torch.arange(n, dtype=F64, device="cuda") * K / (n - 1)
    prev, tot = torch.zeros_like(b), torch.zeros_like(b)
    for e in brk:
        top = torch.sqrt((e * e - b * b).clamp_min(0))
        t = 0.5 * (top - prev)[:, None] * gx + 0.5 * (top + prev)[:, None]
        f, _ = _kernel(kernel, torch.sqrt(b[:, None] ** 2 + t * t))
        tot += (0.5 * (top - prev)[:, None] * gw * f).sum(1)
        prev = top
    tot[-1] = 0
    return 2 * NORM3[kernel] * tot


def _line_fields(c, o, d, x, m, h, rho, cols, spec):
    """Line-integrated sums (scatter), with the tabulated and linearly interpolated integral."""
    K, ns = SUPPORT[c["kernel"]], o[0].numel()
    lut = _line_table(c["kernel"])
    dq = K / (lut.numel() - 1)
    mr = m / rho
    S1 = torch.zeros(ns, dtype=F64, device="cuda")
    Sw = torch.zeros(len(cols), ns, dtype=F64, device="cuda")
    for at in torch.split(torch.arange(ns, device="cuda"), max(1, (1 << 25) // x[0].numel())):
        D = [x[k][None, :] - o[k][at][:, None] for k in range(3)]
        t = sum(D[k] * d[k][at][:, None] for k in range(3))
        s2 = (sum(v * v for v in D) - t * t).clamp_min(0)
        i, j = torch.nonzero(s2 <= (K * h)[None, :] ** 2, as_tuple=True)
        u = torch.sqrt(s2[i, j]) / h[j] / dq
        k = u.long().clamp_max(lut.numel() - 2)
        W = torch.where(u < lut.numel() - 1, torch.lerp(lut[k], lut[k + 1], u - k), torch.zeros_like(u)) / h[j]
        S1.index_add_(0, at[i], mr[j] * W)
        for q, A in enumerate(cols):
            Sw[q].index_add_(0, at[i], A[j] * mr[j] * W)
    S1 = torch.where(S1 == 0, torch.full_like(S1, math.nan), S1)
    return [Sw[q] / S1 if n else Sw[q] + 0 * S1 for q, n in zip(spec["scalars"], spec["shepard"])]


def _sample_points(c, seed):
    if "ns" in c:
        return [_scatter_points(c, c["ns"], seed)]
    dt = np.float32 if c["model"] == "disc" else np.float64
    ax = [torch.from_numpy(a).cuda() for a in _axes(c, dt)]
    Z, Y, X = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    out = [[t.reshape(-1).double() for t in (X, Y, Z)]]
    if c.get("box"):
        fr, pr = (torch.from_numpy(v).cuda() for v in _box(seed))
        t = torch.arange(c["box"], device="cuda").to(fr.dtype)
        a = [pr[2 * k] + t * ((pr[2 * k + 1] - pr[2 * k]) / (c["box"] - 1)) for k in range(3)]
        Z, Y, X = torch.meshgrid(a[2], a[1], a[0], indexing="ij")
        out.append([(fr[k] + X * fr[3 + k] + Y * fr[6 + k] + Z * fr[9 + k]).reshape(-1).double() for k in range(3)])
    return out


def _adjoint(c, s, p, gout, spec):
    """Gradients of sum <gout, fields> for m, x and the columns, from the sums' own derivatives (autograd)."""
    K, st = SUPPORT[c["kernel"]], c["strategy"]
    x, h, rho = [p[k] for k in "xyz"], p["h"], p["rho"]
    cols, nc = p["cols"], len(p["cols"])
    ha = _nearest_h(s, x, h) if st != "scatter" else torch.ones_like(s[0])
    tot = {k: torch.zeros_like(p["m"]) for k in ("m", "x", "y", "z")}
    totc = [torch.zeros_like(p["m"]) for _ in cols]
    for g in _groups(s, 16384):  # whole samples: every pair of a sample is in its group
        sg, hg = [t[g] for t in s], ha[g]
        ij = list(_pairs(sg, hg if st != "scatter" else None, x, h, K, st))
        if not ij:
            continue
        i, j = torch.cat([a for a, _ in ij]), torch.cat([b for _, b in ij])
        v = [t[j].clone().requires_grad_(True) for t in (*x, p["m"], *cols)]
        d = [sg[k][i] - v[k] for k in range(3)]
        W, gw = _weights_ad(c["kernel"], d, hg[i], h[j], st)
        w, e = v[3] / rho[j] * W, v[3] / rho[j] * gw
        add = lambda t: torch.zeros(g.numel(), dtype=F64, device="cuda").index_add(0, i, t)  # noqa: E731
        S1 = add(w)
        ok = S1 != 0
        S1 = torch.where(ok, S1, torch.ones_like(S1))
        Sw = [add(v[4 + q] * w) for q in range(nc)]
        out = [Sw[q] / S1 if n else Sw[q] for q, n in zip(spec["scalars"], spec["shepard"])]
        if "grads" in spec:
            G = [add(e * d[k]) for k in range(3)]
            D = [[add(v[4 + q] * e * d[k]) - G[k] * Sw[q] / S1 for k in range(3)] for q in range(nc)]
            out += [D[q][k] for q in spec["grads"] for k in range(3)]
            a, b, f = spec["curls"]
            out += [D[a][0] + D[b][1] + D[f][2], D[f][1] - D[b][2], D[a][2] - D[f][0], D[b][0] - D[a][1]]
        loss = sum((torch.where(ok, o, torch.zeros_like(o)) * go[g]).sum() for o, go in zip(out, gout))
        dv = torch.autograd.grad(loss, v, allow_unused=True)
        for key, t in zip(("x", "y", "z", "m"), dv):
            if t is not None:
                tot[key].index_add_(0, j, t)
        for q in range(nc):
            if dv[4 + q] is not None:
                totc[q].index_add_(0, j, dv[4 + q])
    return dict(m=tot["m"], x=tot["x"], y=tot["y"], z=tot["z"], cols=totc)


def _weights_ad(kernel, d, ha, hb, strategy):
    r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
    off = (r2 == 0).to(r2.dtype)  # keeps sqrt differentiable at a sample on its particle
    return _weights(kernel, [d[0] + 1e-30 * off, d[1], d[2]], ha, hb, strategy)


def exact(case, seed):
    c = dict(case)
    kind, n = c["kind"], c["n"]
    if kind in ("beam", "train"):  # lines times particles without a tree: minutes
        return None
    p = _particles(c, seed)
    x = [p[k].double() for k in "xyz"]
    m, h, rho = (p[k].double() for k in ("m", "h", "rho"))
    cols = [t.double() for t in p["cols"]]
    if kind == "density":
        K, st = SUPPORT[c["kernel"]], c["strategy"]
        out = torch.zeros_like(m)
        for i, j in _pairs(x, h, x, h, K, st):
            W, _ = _weights(c["kernel"], [t[i] - t[j] for t in x], h[i], h[j], st)
            out.index_add_(0, i, m[j] * W)
        return out
    spec = CATALOGS[c["cat"]]
    if kind == "lines":
        return _line_fields(c, *_sight_lines(c, seed), x, m, h, rho, cols, spec)
    if kind == "adjoint":
        ns = c.get("ns") or c["nx"] * c["ny"] * c["nz"]
        g = _gen(seed, 4)
        gout = [_randn(g, ns) for _ in range(P.CatalogC(**spec).L)]
        return _adjoint(c, _sample_points(c, seed)[0], p, gout, spec)
    return [f for s in _sample_points(c, seed) for f in _fields(c, s, x, m, h, rho, cols, spec)]
