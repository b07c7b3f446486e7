"""Performance cases of the hydrodynamic step, through the public Python entry points.

A hydro pass is what a driver does between two outputs: the state goes in from page-locked host
memory (``Context.upload``), a number of steps run, the state comes back (``download``) with the
clock.  Initial states are made on the GPU from the seed: the workloads of
``tlaloque_gb300/problems.py`` with seeded parameters and a perturbed medium.  ``exact`` restates
the step in plain torch FP64 (source citations in ``tlaloque_gb300/csrc/tlq_physics.cuh``).
"""
from __future__ import annotations

import math

import numpy as np
import torch

AMU, KB, GR = 1.660538782e-24, 1.380650400e-16, 6.67430e-8
PC, YEAR, MSUN, KMS = 3.085677588e18, 3.155673600e7, 1.988920000e33, 1.0e5
MU = 1.3
T_FLOOR = 10.0
OUTFLOW, REFLECTIVE, PERIODIC = 1, 2, 3
LIMITERS = {"vanleer": 2, "minmod": 3}
SOLVERS = {"hllc": 0, "hll": 1}
COOLINGS = {"none": 0, "ref": 1, "subcycle": 2, "mlp": 3, "exact": 4}
MLP_BOX = (-4.0, 4.0, 4.0, 8.5, -8.0, 1.0)  # tlq_surrogate_opts_default
MEMBERS = (128, 48, 96, 64, 64, 128, 48, 96)


def _case(name, problem, n, precision, steps, **kw):
    c = {"problem": problem, "n": n, "precision": precision, "cooling": "none", "limiter": "vanleer", "solver": "hllc",
         "steps": steps, "by_step": False, "tuned": False}
    c.update(kw)
    return {"name": name, **c} if name else c


def listed():
    return [
        # the Sod tube of the validation runs, driven like the Fortran loop: one call and one clock
        # read per step; the smallest mesh, where latency and launches count
        _case("sod_256x4x4_fp64", "sod", 256, "fp64", 16, solver="hll", by_step=True),
        # the smallest bubble of the ensemble's sizes as a single run, stepped one call at a time
        _case("wind_48_mixed", "wind", 48, "mixed", 16, cooling="subcycle", by_step=True),
        # the 3-D Sedov blast of the validation runs in the default (reference-exact) arithmetic
        _case("sedov_128_fp64", "sedov", 128, "fp64", 4),
        # the reference's own diagonal Sod test at its own size, not a multiple of the tile
        _case("diagsod_150_mixed", "diagsod", 150, "mixed", 16),
        # the headline bubble in the default arithmetic: cooling, wind, point mass
        _case("wind_256_fp64", "wind", 256, "fp64", 2, cooling="subcycle"),
        # the headline bubble in mixed precision, tuned once as a long run would be
        _case("wind_256_mixed", "wind", 256, "mixed", 16, cooling="subcycle", tuned=True),
        # a host that keeps the state and takes it in and out every step (the drop-in of a driver
        # with its own physics between steps)
        _case("wind_128_roundtrip", "wind", 128, "mixed", 1, cooling="exact", by_step=True),
        # the radiative clumpy medium with the learned cooling at work
        _case("clumpy_256_mlp", "clumpy", 256, "mixed", 8, cooling="mlp", tuned=True),
        # the self-gravitating cloud: two multigrid solves a step
        _case("cloud_128_mixed", "cloud", 128, "mixed", 2, multipole=True),
        _case("cloud_64_fp64", "cloud", 64, "fp64", 2, multipole=False),
        # a parameter scan: bubbles of four sizes advanced together, tuned
        _case("ensemble_8", "ensemble", 8, "mixed", 16, cooling="mlp", tuned=True),
        # the surrogate's training direction: loss and gradient of one large batch
        _case("mlp_grad_262144", "mlp_grad", 262144, "fp32", 1),
    ]


def draw(rng):
    kind = rng.choice(["sod", "sedov", "diagsod", "wind", "wind", "clumpy", "cloud", "box", "box", "ensemble", "mlp_grad"])
    if kind == "mlp_grad":
        return _case("", kind, int(round(math.exp(rng.uniform(math.log(1000), math.log(262144))))), "fp32", 1)
    if kind == "cloud":
        mixed = rng.random() < 0.5
        return _case("", kind, rng.choice([16, 32, 64, 128]), "mixed" if mixed else "fp64", rng.randint(1, 2),
                     multipole=rng.random() < 0.5, by_step=rng.random() < 0.3)
    if kind == "ensemble":
        return _case("", kind, rng.randint(2, 8), "mixed", rng.randint(4, 16), cooling=rng.choice(["subcycle", "exact", "mlp"]),
                     tuned=rng.random() < 0.5)
    mixed = rng.random() < 0.5
    n = int(round(math.exp(rng.uniform(math.log(24), math.log(240 if mixed else 160)))))
    if kind == "sod":
        n = int(round(math.exp(rng.uniform(math.log(64), math.log(2000)))))
    if kind == "wind":
        n += n % 2  # the star sits on a cell corner: at the centre of a cell its wind has no finite density
    cells = n * 16 if kind == "sod" else n**3
    most = (100_000_000 if mixed else 12_000_000) // cells
    kw = {"tuned": rng.random() < 0.3, "by_step": rng.random() < 0.4}
    if kind in ("wind", "clumpy"):
        kw["cooling"] = rng.choice(["none", "ref", "subcycle", "exact"] + (["mlp"] if mixed else []))
    if kind in ("box", "sod"):
        kw["solver"] = rng.choice(["hllc", "hll"])
    if kind == "box":
        kw["limiter"] = rng.choice(["vanleer", "vanleer", "minmod"])
        kw["bc"] = rng.randint(0, 3)
    return _case("", kind, n, "mixed" if mixed else "fp64", max(1, min(16, rng.randint(1, 16), most)), **kw)


# ---- states --------------------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Rng:
    """Seeded numbers: scalars from the host generator, fields from the device's."""

    def __init__(self, seed):
        self.host = np.random.default_rng(seed)
        self.dev = torch.Generator(_device()).manual_seed(int(seed) * 7919 + 1)

    def uniform(self, lo, hi):
        return float(self.host.uniform(lo, hi))

    def normal(self, shape):
        return torch.randn(shape, generator=self.dev, device=_device(), dtype=torch.float64)


def _spec(n3, lo, hi, case, **kw):
    s = {"n": n3, "lo": lo, "hi": hi, "gamma": 5.0 / 3.0, "cfl": 0.4, "eta": 0.5e-2, "mu0": 1.0, "bc": (OUTFLOW,) * 6,
         "cooling": case["cooling"], "limiter": case["limiter"], "solver": case["solver"], "sub_frac": 0.1,
         "max_sub": 16, "cooling_limit": 0.5, "winds": [], "masses": [], "T": None, "logL": None, "grav": None}
    s.update(kw)
    if s["cooling"] in ("exact", "mlp"):
        s["sub_frac"] = 2e-3
    return s


def _dx(s):
    return [(s["hi"][q] - s["lo"][q]) / s["n"][q] for q in range(3)]


def _centres(s):
    """x, y, z of the cells -1..n+2, shaped to broadcast over (z, y, x)."""
    out = []
    for q in range(3):
        i = torch.arange(-1, s["n"][q] + 3, device=_device(), dtype=torch.float64)
        d = _dx(s)[q]
        v = (s["lo"][q] + d * i) - d / 2.0
        out.append(v.reshape([-1 if a == 2 - q else 1 for a in range(3)]))
    return out


def _conserved(s, rho, v, p):
    shape = tuple(m + 4 for m in reversed(s["n"]))
    rho, p = (torch.as_tensor(a, dtype=torch.float64, device=_device()).expand(shape) for a in (rho, p))
    v = [torch.as_tensor(a, dtype=torch.float64, device=_device()).expand(shape) for a in v]
    k2 = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
    return torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], 0.5 * rho * k2 + p / (s["gamma"] - 1.0)])


def _gaussian(r, n, slope=-5.0 / 3.0):
    """Periodic Gaussian field on n^3, unit variance, shell spectrum k^slope, with two wrapped ghost layers."""
    k = torch.fft.fftfreq(n, 1.0 / n, device=_device(), dtype=torch.float64)
    kz = torch.fft.rfftfreq(n, 1.0 / n, device=_device(), dtype=torch.float64)
    kk = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2)
    kk[0, 0, 0] = 1.0
    amp = kk ** ((slope - 2.0) / 2.0)
    amp[0, 0, 0] = 0.0
    f = torch.fft.irfftn(amp * torch.fft.rfftn(r.normal((n, n, n))), s=(n, n, n))
    f = (f - f.mean()) / f.std()
    g = torch.arange(-2, n + 2, device=_device()) % n
    return f[g][:, g][:, :, g]


def _cooling_table():
    """problems.synthetic_cooling_table: 200 nodes, 1e4-1e8 K, peak 10^-21.5 at 2e5 K."""
    T = np.logspace(4.0, 8.0, 200)
    lt = np.log10(T)
    pk, ltp = -21.5, math.log10(2e5)
    s_lo = (pk + 23.12) / (ltp - 4.0)
    l7 = pk - 0.7 * (7.0 - ltp)
    return T, np.where(lt < ltp, pk + s_lo * (lt - ltp), np.where(lt <= 7.0, pk - 0.7 * (lt - ltp), l7 + 0.5 * (lt - 7.0)))


def _wind(case, n, r):
    L = 8.0 * PC
    T, logL = _cooling_table()
    s = _spec((n, n, n), (-L / 2,) * 3, (L / 2,) * 3, case, mu0=MU, T=T, logL=logL,
              masses=[(0.0, 0.0, 0.0, 10.0 * MSUN)])
    nd = math.exp(r.uniform(math.log(0.3), math.log(3.0)))
    s["winds"] = [{"radius": 4.0 * _dx(s)[0], "mdot": 1e-6 * MSUN / YEAR, "vinf": r.uniform(800.0, 2500.0) * KMS,
                   "temp": 1e4, "mu": MU}]
    rho = nd * MU * AMU * (1.0 + 0.01 * r.normal((n + 4,) * 3).clamp(-4, 4))
    return s, _conserved(s, rho, (0.0, 0.0, 0.0), nd * KB * 1.05e4)


def _hydro(case, seed):
    """(spec, U0): U0 (5, z, y, x) with every cell set, ghosts included."""
    r, n, kind = _Rng(seed), case["n"], case["problem"]
    if kind == "wind":
        return _wind(case, n, r)
    if kind == "sod":
        d = 1.0 / n
        s = _spec((n, 4, 4), (0.0,) * 3, (1.0, 4 * d, 4 * d), case, gamma=1.4)
        left = _centres(s)[0] < r.uniform(0.4, 0.6)
        rho = torch.where(left, r.uniform(0.9, 1.1), r.uniform(0.1, 0.15))
        return s, _conserved(s, rho, (0.0, 0.0, 0.0), torch.where(left, 1.0, r.uniform(0.08, 0.12)))
    if kind == "diagsod":
        s = _spec((n, n, n), (-0.25,) * 3, (0.25,) * 3, case, cfl=0.8, eta=0.05)
        x, y, z = _centres(s)
        left = -x - y - z > r.uniform(-0.05, 0.05)
        return s, _conserved(s, torch.where(left, r.uniform(3.8, 4.2), 1.0), (0.0, 0.0, 0.0), torch.where(left, 1.0, 0.1795))
    if kind == "sedov":
        s = _spec((n, n, n), (-0.5,) * 3, (0.5,) * 3, case, cfl=0.3)
        x, y, z = _centres(s)
        rr = torch.sqrt(x * x + y * y + z * z)
        hot = r.uniform(0.8, 1.2) * 2.0 / 3.0 / (4.0 / 3.0 * math.pi * (3.0 * _dx(s)[0]) ** 3)
        rho = 1.0 + 0.01 * r.normal(rr.shape).clamp(-4, 4)
        return s, _conserved(s, rho, (0.0, 0.0, 0.0), torch.where(rr < 3.0 * _dx(s)[0], hot, 1e-5))
    if kind == "clumpy":
        L = 8.0 * PC
        T, logL = _cooling_table()
        s = _spec((n, n, n), (-L / 2,) * 3, (L / 2,) * 3, case, mu0=MU, T=T, logL=logL, bc=(PERIODIC,) * 6)
        nd = torch.exp(_gaussian(r, n))
        nd = nd / nd.mean()
        lgT = 3.0 + 5.0 * torch.special.ndtr(_gaussian(r, n))
        v = [2.0 * math.sqrt(s["gamma"] * KB * 1e4 / (MU * AMU) / 3.0) * _gaussian(r, n) for _ in range(3)]
        return s, _conserved(s, nd * MU * AMU, v, nd * KB * 10.0**lgT)
    if kind == "cloud":
        L = 4.0 * PC
        s = _spec((n, n, n), (-L / 2,) * 3, (L / 2,) * 3, case, mu0=MU, grav=int(case["multipole"]))
        x, y, z = _centres(s)
        rr = torch.sqrt(x * x + y * y + z * z)
        nd = r.uniform(400.0, 600.0)
        rho = torch.where(rr < r.uniform(0.8, 1.2) * PC, 1.0 + 0.01 * r.normal(rr.shape).clamp(-4, 4), 0.01)
        return s, _conserved(s, nd * MU * AMU * rho, (0.0, 0.0, 0.0), nd * KB * 50.0)
    # box: a smooth random flow on an uneven mesh with one of four sets of boundaries
    n3 = (n, max(2, int(n * 0.6)), max(2, int(n * 0.75)))
    bc = [(OUTFLOW,) * 6, (PERIODIC,) * 6, (REFLECTIVE,) * 6,
          (REFLECTIVE, OUTFLOW, PERIODIC, PERIODIC, OUTFLOW, REFLECTIVE)][case["bc"]]
    s = _spec(n3, (0.0,) * 3, (1.0, 0.6, 0.75), case, bc=bc)
    x, y, z = _centres(s)
    f = []
    for _ in range(5):
        a = 0.0
        for q in range(4):
            k = [2.0 * math.pi * int(r.host.integers(1, 5)) / s["hi"][w] for w in range(3)]
            a = a + 0.25 * torch.cos(k[0] * x + r.uniform(0, 6)) * torch.cos(k[1] * y + r.uniform(0, 6)) * torch.cos(
                k[2] * z + r.uniform(0, 6))
        f.append(a)
    return s, _conserved(s, torch.exp(0.5 * f[0]), (f[2], f[3], f[4]), torch.exp(0.5 * f[1]))


def _members(case, seed):
    return [_wind(case, n, _Rng(seed * 64 + q)) for q, n in enumerate(MEMBERS[: case["n"]])]


def _network(seed):
    """Weights as a stored network has them (Glorot range, a small output layer)."""
    g = np.random.default_rng(seed)
    a = math.sqrt(6.0 / 128)
    w = [g.uniform(-0.3, 0.3, 192), g.uniform(-0.1, 0.1, 64), g.uniform(-a, a, 4096), g.uniform(-0.1, 0.1, 64),
         g.uniform(-a, a, 4096), g.uniform(-0.1, 0.1, 64), 0.1 * g.uniform(-0.3, 0.3, 64), np.zeros(1)]
    return np.concatenate(w).astype(np.float32)


def _samples(case, seed):
    g = np.random.default_rng(seed)
    X = g.uniform(-1.0, 1.0, (case["n"], 3)).astype(np.float32)
    Y = (0.5 * np.sin(2.0 * X[:, 0]) + X[:, 1] * X[:, 2] - 0.3).astype(np.float32)
    return _network(seed + 1), X, Y


# ---- the measured path ---------------------------------------------------------------------------
def _config(s, precision):
    from tlaloque_gb300 import tlq

    cfg = tlq.Config(nx=s["n"][0], ny=s["n"][1], nz=s["n"][2], xl=s["lo"][0], xr=s["hi"][0], yl=s["lo"][1],
                     yr=s["hi"][1], zl=s["lo"][2], zr=s["hi"][2], gamma=s["gamma"], cfl=s["cfl"], eta=s["eta"],
                     mu0=s["mu0"], cooling_limit=s["cooling_limit"], limiter=LIMITERS[s["limiter"]],
                     solver=SOLVERS[s["solver"]], bc=s["bc"], cooling=COOLINGS[s["cooling"]],
                     cool_max_sub=s["max_sub"], cool_sub_frac=s["sub_frac"],
                     precision=tlq.PREC_MIXED if precision == "mixed" else tlq.PREC_FP64, cool_T=s["T"],
                     cool_logL=s["logL"])
    if s["grav"] is not None:
        cfg.self_gravity, cfg.grav_bc = 1, tlq.GBC_MULTIPOLE if s["grav"] else tlq.GBC_ZERO
    cfg.winds = [tlq.Wind(**w) for w in s["winds"]]
    if s["masses"]:
        cfg.masses = np.array(s["masses"])
    return cfg


def _host(cfg):
    """A page-locked host array in the reference layout."""
    flat = torch.empty(int(np.prod(cfg.shape)), dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return flat, flat.numpy().reshape(cfg.shape, order="F")


def _load(ctx, U0):
    """The host state (after borders, mainHD.f90:38) and the array the results come back to."""
    flat, U = _host(ctx.cfg)
    flat.copy_(U0.permute(1, 2, 3, 0).reshape(-1))
    ctx.borders(U, 1)
    back, out = _host(ctx.cfg)
    ctx.upload(U)
    return {"U": U, "out": out, "keep": (flat, back)}


def _surrogate(ctx):
    if ctx.cfg.cooling == COOLINGS["mlp"]:
        half = [(MLP_BOX[2 * q] + MLP_BOX[2 * q + 1]) / 2 if w == 0 else (MLP_BOX[2 * q + 1] - MLP_BOX[2 * q]) / 2
                for q in range(3) for w in range(2)]
        ctx.set_cooling_surrogate(_network(5), half, MLP_BOX)


def prepare(case, seed):
    from tlaloque_gb300 import tlq

    if case["problem"] == "mlp_grad":
        return {"case": case, "args": _samples(case, seed)}
    if case["problem"] == "ensemble":
        ms = _members(case, seed)
        batch = tlq.Batch([_config(s, "mixed") for s, _ in ms])
        loads = []
        for ctx, (s, U0) in zip(batch.members, ms):
            _surrogate(ctx)
            loads.append(_load(ctx, U0))
        if case["tuned"]:
            batch.autotune()
        return {"case": case, "batch": batch, "loads": loads}
    s, U0 = _hydro(case, seed)
    ctx = tlq.Context(_config(s, case["precision"]))
    _surrogate(ctx)
    load = _load(ctx, U0)
    if case["tuned"]:
        ctx.autotune()
    return {"case": case, "ctx": ctx, **load}


def _result(U, t, dt):
    """The interior of the state and the clock (the second ghost layer and the edges are not the step's)."""
    V = U[:, 2:-2, 2:-2, 2:-2]
    return {"density": V[0], "momentum": V[1:4], "energy": V[4], "t": t, "dt": dt}


def run(state):
    case = state["case"]
    if case["problem"] == "mlp_grad":
        from tlaloque_gb300 import tlq

        loss, grad = tlq.mlp_loss_grad(*state["args"])
        return {"loss": loss, "grad": grad}
    if case["problem"] == "ensemble":
        batch = state["batch"]
        for ctx, l in zip(batch.members, state["loads"]):
            ctx.upload(l["U"])
        batch.run(case["steps"])
        out = []
        for ctx, l in zip(batch.members, state["loads"]):
            ctx.download(l["out"])
            t, _, dt, _ = ctx.time()
            out.append(_result(l["out"], t, dt))
        return out
    ctx = state["ctx"]
    ctx.upload(state["U"])
    if case["by_step"]:
        for _ in range(case["steps"]):
            t, _, dt = ctx.step()
    else:
        ctx.advance(case["steps"])
        t, _, dt, _ = ctx.time()
    ctx.download(state["out"])
    return _result(state["out"], t, dt)


def work(case):
    """The state in from the host and back (40 B a cell each), and per step the state read and written
    once; operations per zone-update as the oracle's counting build has them, for self-gravity 10
    V-cycles of ~100 operations a cell in each step."""
    n, kind = case["n"], case["problem"]
    if kind == "mlp_grad":
        return {"bytes": n * 16 + 2 * 4 * 8641, "flops": n * 6.0 * 8448}
    cells = sum(m**3 for m in MEMBERS[:n]) if kind == "ensemble" else (
        16 * n if kind == "sod" else n * int(n * 0.6) * int(n * 0.75) if kind == "box" else n**3)
    per = {"sod": 1338, "wind": 1023, "clumpy": 1023, "ensemble": 1023, "cloud": 775 + 1000}.get(kind, 775)
    return {"bytes": cells * 80.0 * (1 + case["steps"]), "flops": float(cells) * case["steps"] * per}


# ---- 64-bit restatement --------------------------------------------------------------------------
def _borders(s, U, layers):
    """boundariesI/II of a single rank, then the winds (boundaries.f90:183-257, :433-531)."""
    for q in range(3):
        a, n = 3 - q, s["n"][q]
        at = lambda i: U.select(a, i + 1)  # noqa: E731
        for side in range(2):
            kind = s["bc"][2 * q + side]
            near, far, out = (n, 1, 1) if side else (1, n, -1)
            for l in range(layers):
                dst = (n + 1 if side else 0) + out * l
                if kind == PERIODIC:
                    v = at(far + out * l).clone()
                else:
                    v = at(near - (out * l if kind == REFLECTIVE else 0)).clone()
                    if kind == REFLECTIVE:
                        v[q + 1] = -v[q + 1]
                at(dst).copy_(v)
    for w in s["winds"]:
        x, y, z = _centres(s)
        d = torch.sqrt(x * x + y * y + z * z)
        m = d < w["radius"]
        x, y, z = (c.expand(d.shape)[m] for c in (x, y, z))
        d = d[m]
        rho = w["mdot"] / (w["vinf"] * d * d * 4.0 * 3.14159265358979)
        U[0][m] = rho
        for e, c in enumerate((x, y, z)):
            U[1 + e][m] = rho * w["vinf"] * c / d
        U[4][m] = 0.5 * rho * w["vinf"] ** 2 + rho * KB * w["temp"] / (w["mu"] * AMU) / (s["gamma"] - 1.0)


def _prims(s, U):
    v = U[1:4] / U[0]
    p = (s["gamma"] - 1.0) * (U[4] - 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / U[0])
    return torch.cat([U[:1], v, p.clamp_min(1e-20)[None]])


def _average(a, b, lim):
    if lim == "vanleer":
        ab = a * b
        ok = ab > 0
        return torch.where(ok, ab * (a + b) / torch.where(ok, a * a + b * b, 1.0), 0.0)
    sg = torch.copysign(torch.ones_like(a), a)
    return sg * torch.minimum(a.abs(), sg * b).clamp_min(0.0)


def _flux(s, w, d):
    un = w[d]
    f = w[0] * un * w
    f[0] = w[0] * un
    f[d] = f[d] + w[4]
    f[4] = un * (0.5 * w[0] * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2) + s["gamma"] / (s["gamma"] - 1.0) * w[4])
    return f


def _faces(s, U, W, d, second):
    """Fluxes at the n+1 faces of direction d (1..3) of the interior's columns (HLLC.f90, HLL.f90)."""
    a, n = 4 - d, s["n"][d - 1]
    for b in range(1, 4):
        if b != a:
            U, W = U.narrow(b, 2, U.shape[b] - 4), W.narrow(b, 2, W.shape[b] - 4)
    cut = lambda v, i: v.narrow(a, i, n + 1)  # noqa: E731
    wl, wr, ul, ur = cut(W, 1), cut(W, 2), cut(U, 1), cut(U, 2)
    if second:
        dm = wr - wl
        wl, wr = (wl + 0.5 * _average(wl - cut(W, 0), dm, s["limiter"]),
                  wr - 0.5 * _average(dm, cut(W, 3) - wr, s["limiter"]))
    g = s["gamma"]
    cl, cr = torch.sqrt(g * wl[4] / wl[0]), torch.sqrt(g * wr[4] / wr[0])
    sl, sr = torch.minimum(wl[d] - cl, wr[d] - cr), torch.maximum(wl[d] + cl, wr[d] + cr)
    if s["solver"] == "hll":
        fl, fr = _flux(s, wl, d), _flux(s, wr, d)
        return torch.where(sl >= 0, fl, torch.where(sr <= 0, fr, (sr * fl - sl * fr + sl * sr * (ur - ul)) / (sr - sl)))
    al, ar = wl[0] * (sl - wl[d]), wr[0] * (sr - wr[d])
    sst = (wr[4] - wl[4] + al * wl[d] - ar * wr[d]) / (al - ar)
    left = (sl >= 0) | ((sr > 0) & (sst >= 0))
    star = (sl < 0) & (sr > 0)
    w, u, sk, ak = torch.where(left, wl, wr), torch.where(left, ul, ur), torch.where(left, sl, sr), torch.where(left, al, ar)
    f = _flux(s, w, d)
    rs = ak / (sk - sst)
    us = rs * w
    us[0] = rs
    us[d] = rs * sst
    us[4] = rs * (u[4] / w[0] + (sst - w[d]) * (sst + w[4] / ak))
    return torch.where(star, f + sk * (us - u), f)


def _inside(v):
    return v[..., 2:-2, 2:-2, 2:-2]


def _godunov(s, old, U, W, dt, second, dphi):
    out = old.clone()
    new = _inside(old).clone()
    for d in (1, 2, 3):
        F = _faces(s, U, W, d, second)
        n = s["n"][d - 1]
        new -= dt / _dx(s)[d - 1] * (F.narrow(4 - d, 1, n) - F.narrow(4 - d, 0, n))
    if dphi is not None:
        w = _inside(W)
        for q in range(3):
            new[1 + q] -= dt * w[0] * dphi[q]
            new[4] -= dt * w[0] * w[1 + q] * dphi[q]
    _inside(out).copy_(new)
    return out


def _potential(s):
    if not s["masses"]:
        return None
    x, y, z = _centres(s)
    phi = 0.0
    for m in s["masses"]:
        phi = phi - GR * m[3] / torch.sqrt((m[0] - x) ** 2 + (m[1] - y) ** 2 + (m[2] - z) ** 2)
    d, n = _dx(s), s["n"]
    mid = [slice(2, 2 + n[q]) for q in (2, 1, 0)]
    out = []
    for q in range(3):
        hi, lo = list(mid), list(mid)
        hi[2 - q], lo[2 - q] = slice(3, 3 + n[q]), slice(1, 1 + n[q])
        out.append((phi[tuple(hi)] - phi[tuple(lo)]) / (2.0 * d[q]))
    return out


def _coef(t, temp):
    T, lT, C = t
    i = torch.searchsorted(T, temp, right=True).clamp(1, len(T) - 1)
    v = (C[i] - C[i - 1]) / (lT[i] - lT[i - 1]) * (torch.log10(temp) - lT[i - 1]) + C[i - 1]
    return 10.0 ** torch.where(temp >= T[-1], C[-1], v)


def _exact_drop(t, temp, lam, tau):
    """The temperature after exact cooling by tau (a piecewise power-law table, Townsend 2009)."""
    T, lT, C = t
    n = len(T)
    sl = torch.cat([(C[1:] - C[:-1]) / (lT[1:] - lT[:-1]), torch.zeros(1, dtype=C.dtype, device=C.device)])
    a = 1.0 - sl
    flat = a.abs() < 1e-9
    G = torch.where(flat[:-1], torch.log(T[1:] / T[:-1]), ((T[1:] / T[:-1]) ** a[:-1] - 1.0) / torch.where(flat, 1.0, a)[:-1])
    G = torch.cat([torch.zeros(1, dtype=C.dtype, device=C.device), torch.cumsum(T[:-1] / 10.0 ** C[:-1] * G, 0)])
    i = torch.searchsorted(T, temp, right=True).clamp(1, n) - 1
    ai, fi = torch.where(flat[i], 1.0, a[i]), flat[i]
    ti = torch.where(fi, -torch.log(T[i] / temp), (1.0 - (T[i] / temp) ** ai) / ai)
    stay = temp * torch.where(fi, torch.exp(-tau), (1.0 - ai * tau).clamp_min(0.0) ** (1.0 / ai))
    left = G[i] - (tau - ti) * temp / lam
    j = (torch.searchsorted(G, left, right=True) - 1).clamp(0, n - 1)
    j = torch.minimum(j, (i - 1).clamp_min(0))
    q = (left - G[j]) * 10.0 ** C[j] / T[j]
    aj = torch.where(flat[j], 1.0, a[j])
    moved = T[j] * torch.where(flat[j], torch.exp(q), (1.0 + aj * q).clamp_min(0.0) ** (1.0 / aj))
    return torch.where(tau <= ti, stay, torch.where(left > 0, moved, T[0]))


def _cool(s, U, dt):
    if s["cooling"] == "none":
        return
    t = [torch.as_tensor(v, device=U.device, dtype=torch.float64) for v in (s["T"], np.log10(s["T"]), s["logL"])]
    V = _inside(U)
    w = _prims(s, V)
    rho, p = w[0], w[4]
    kT, gm1 = s["mu0"] * AMU / KB, s["gamma"] - 1.0
    nd = rho / (s["mu0"] * AMU)
    temp = p / rho * kT
    on = temp >= t[0][0]
    safe = torch.where(on, temp, t[0][0])
    ce = _coef(t, safe) * nd * nd / (p / gm1)
    tau = ce * dt
    sub = on & (tau > s["sub_frac"]) if s["cooling"] != "ref" else torch.zeros_like(on)
    nsub = torch.ones_like(tau)
    if s["cooling"] == "subcycle":
        nsub = torch.where(sub, torch.ceil(tau / s["sub_frac"]).clamp(1, s["max_sub"]), nsub)
    live, pn = on.clone(), p.clone()
    for q in range(int(nsub.max())):
        live = live & (q < nsub)
        if q:
            temp = pn / rho * kT
            live = live & (temp >= t[0][0])
            ce = _coef(t, torch.where(live, temp, t[0][0])) * nd * nd / (pn / gm1)
        f = torch.exp(-ce * dt / nsub).clamp_min(1.0 - s["cooling_limit"])
        low = temp * f < T_FLOOR
        f = torch.where(low, T_FLOOR / temp, f)
        pn = torch.where(live, pn * f, pn)
        live = live & ~low
    if s["cooling"] in ("exact", "mlp"):
        temp = p / rho * kT
        T1 = _exact_drop(t, torch.where(sub, temp, 2 * t[0][0]), _coef(t, torch.where(sub, temp, 2 * t[0][0])), tau)
        pn = torch.where(sub, p * T1 / temp, pn)
    V[4] += (pn - p) / gm1


def _steps(s, U, steps):
    U = U.clone()
    _borders(s, U, 1)
    dphi = _potential(s)
    tt, dt = 0.0, 0.0
    for _ in range(steps):
        W = _prims(s, U)
        w = _inside(W)
        cs = torch.sqrt(s["gamma"] * w[4] / w[0])
        dt = s["cfl"] * min(_dx(s)[q] / float((w[1 + q].abs() + cs).max()) for q in range(3)) / math.sqrt(3.0)
        P = _godunov(s, U, U, W, dt / 2.0, False, dphi)
        _borders(s, P, 2)
        new = _godunov(s, U, P, _prims(s, P), dt, True, dphi)
        _borders(s, new, 1)
        lap = -6.0 * _inside(U)
        for a in (1, 2, 3):
            for off in (1, 3):
                v = U
                for b in (1, 2, 3):
                    v = v.narrow(b, off if b == a else 2, U.shape[b] - 4)
                lap += v
        _inside(new).add_(lap, alpha=s["eta"])
        U = new
        _cool(s, U, dt)
        tt += dt
    V = _inside(U).permute(0, 3, 2, 1)
    return {"density": V[0], "momentum": V[1:4], "energy": V[4], "t": tt, "dt": dt}


def _exact_grad(case, seed):
    P, X, Y = (torch.as_tensor(v, dtype=torch.float64, device=_device()) for v in _samples(case, seed))
    P.requires_grad_(True)
    at, parts = 0, []
    for shape in ((64, 3), (64,), (64, 64), (64,), (64, 64), (64,), (64,), (1,)):
        parts.append(P[at : at + math.prod(shape)].reshape(shape))
        at += math.prod(shape)
    h = X
    for q in range(3):
        h = torch.nn.functional.silu(h @ parts[2 * q].T + parts[2 * q + 1])
    loss = ((h @ parts[6] + parts[7] - Y) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": P.grad}


def exact(case, seed):
    if case["problem"] == "mlp_grad":
        return _exact_grad(case, seed)
    if case["problem"] == "ensemble":
        return [_steps(s, U, case["steps"]) for s, U in _members(case, seed)]
    if case["problem"] == "cloud":
        return None  # the reference's Gauss-Seidel order is sequential: minutes in plain torch
    return _steps(*_hydro(case, seed), case["steps"])
