"""The work that users of this framework have it do, as timed cases.

A pass of a flow or soil case is what a program around the solver repeats
between two outputs: a number of steps of the domain, then the fields it looks
at, read back to the host. The network cases are one training call and one
inference call. Sizes and options come from the benchmark's workloads
(poiseuille2d, dam2d, dam3d, dam3d_coarse, the granular ensemble), the tests
and generic lattices between them.

Initial states are disordered flows, not lattices at rest: free particles
displaced from the lattice, a smooth velocity field with small-scale noise, and
density (fluids) or stress (soil) noise, all from the seed.

The FP32C form sums its pair terms in FP32: what it returns of those sums
(accelerations, rates, and the velocities, densities and stresses they feed) is
taken as FP32; positions, which it integrates in FP64, stay FP64. The FP64
form's fields are all FP64.
"""
import functools
import math

import numpy as np
import torch

from persiansph_gb300 import scenarios
from persiansph_gb300.closure import ClosureNet, default_network_path, les_case
from persiansph_gb300.solver import GpuDomain, GpuEnsemble

FP64, FP32C = 0, 1


def listed():
    return [
        # the smallest call: one step of the 920-particle channel, looked at after it (an interactive
        # or coupled run, where launches and latency are all there is)
        {"name": "channel_one_step", "kind": "channel", "dx": 2.5e-5, "H": 1.0e-3, "W": 0.5e-3, "precision": FP64,
         "scheme": 1, "steps": 1},
        # the same channel over an output interval, FP32C
        {"name": "channel_fp32", "kind": "channel", "dx": 2.5e-5, "H": 1.0e-3, "W": 0.5e-3, "precision": FP32C,
         "scheme": 1, "steps": 40},
        # a coarse 2D dam break of a parameter study: odd sizes, leapfrog, FP64
        {"name": "dam2d_coarse", "kind": "dam2d", "dx": 0.0167, "L": 0.73, "H": 1.31, "TL": 2.9, "TH": 2.2,
         "precision": FP64, "scheme": 1, "steps": 20},
        # the 2D dam break of the benchmark (86k particles) in both forms
        {"name": "dam2d_fp64", "kind": "dam2d", "dx": 0.005, "L": 1.0, "H": 2.0, "TL": 4.0, "TH": 3.0,
         "precision": FP64, "scheme": 0, "steps": 20},
        {"name": "dam2d_fp32", "kind": "dam2d", "dx": 0.005, "L": 1.0, "H": 2.0, "TL": 4.0, "TH": 3.0,
         "precision": FP32C, "scheme": 0, "steps": 40},
        # the 3D dam break in the drop-in FP64 form (177k particles, the closure's coarse lattice)
        {"name": "dam3d_fp64", "kind": "dam3d", "dx": 0.02, "L": 1.2, "H": 0.55, "W": 1.0, "TL": 3.22, "TH": 1.0,
         "precision": FP64, "closure": False, "skin": 0, "steps": 10},
        # the closure's own workload: coarse 3D dam break with LES on, FP32C
        {"name": "dam3d_closure", "kind": "dam3d", "dx": 0.02, "L": 1.2, "H": 0.55, "W": 1.0, "TL": 3.22, "TH": 1.0,
         "precision": FP32C, "closure": True, "skin": 0, "steps": 40},
        # a million particles, FP32C without LES, default settings (lists every step)
        {"name": "dam3d_1m", "kind": "dam3d", "dx": 0.01, "L": 1.2, "H": 0.55, "W": 1.0, "TL": 3.22, "TH": 1.0,
         "precision": FP32C, "closure": False, "skin": 0, "steps": 20},
        # the headline: 6.7M particles, FP32C with the closure, the list skin its autotuner picks
        {"name": "dam3d_headline", "kind": "dam3d", "dx": 0.005, "L": 1.2, "H": 0.55, "W": 1.0, "TL": 3.22, "TH": 1.0,
         "precision": FP32C, "closure": True, "skin": 50, "steps": 40},
        # one granular column in the drop-in FP64 form
        {"name": "column_fp64", "kind": "columns", "dx": 2.0e-3, "n": 1, "aspect0": 1.3, "aspect1": 1.3,
         "precision": FP64, "steps": 10},
        # the batched granular columns (ten columns over the 256-column ensemble's range of heights)
        {"name": "columns_fp32", "kind": "columns", "dx": 1.0e-3, "n": 10, "aspect0": 0.5, "aspect1": 4.0,
         "precision": FP32C, "steps": 20},
        # the closure's network: Adam steps on minibatches, then inference on a filtered flow's samples
        {"name": "closure_train", "kind": "net", "samples": 200000, "batch": 4096, "train_steps": 20},
    ]


def draw(rng):
    def lu(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    kind = rng.choice(["channel", "dam2d", "dam2d", "dam3d", "dam3d", "dam3d", "columns", "columns", "net"])
    prec = rng.choice([FP64, FP32C])
    if kind == "channel":
        dx = lu(1.2e-5, 5.0e-5)
        return {"kind": kind, "dx": dx, "H": 2 * dx * rng.randint(10, 40), "W": dx * rng.randint(16, 80),
                "precision": prec, "scheme": rng.choice([0, 1]), "steps": rng.choice([1, 10, 40])}
    if kind == "dam2d":
        dx = lu(0.005, 0.03)
        H = rng.uniform(0.8, 2.0)
        return {"kind": kind, "dx": dx, "L": rng.uniform(0.5, 1.2), "H": H, "TL": rng.uniform(2.0, 4.0), "TH": 1.5 * H,
                "precision": prec, "scheme": rng.choice([0, 1]), "steps": rng.randint(10, 40)}
    if kind == "dam3d":
        closure = prec == FP32C and rng.random() < 0.5
        return {"kind": kind, "dx": lu(0.009, 0.03) if prec == FP32C else lu(0.016, 0.04), "L": rng.uniform(0.5, 1.2),
                "H": rng.uniform(0.3, 0.6), "W": rng.uniform(0.4, 1.0), "TL": rng.uniform(1.6, 3.22), "TH": 1.0,
                "precision": prec, "closure": closure, "skin": rng.choice([0, 50, 100]) if prec == FP32C else 0,
                "steps": rng.randint(5, 40) if prec == FP32C else rng.randint(2, 10)}
    if kind == "columns":
        n = 1 if prec == FP64 else rng.randint(1, 10)
        a = rng.uniform(0.5, 2.0)
        return {"kind": kind, "dx": lu(1.0e-3, 4.0e-3) if prec == FP32C else lu(1.6e-3, 5.0e-3), "n": n, "aspect0": a,
                "aspect1": 4.0 if n > 1 else a, "precision": prec, "steps": rng.randint(4, 20)}
    return {"kind": kind, "samples": int(lu(5000, 400000)), "batch": rng.randint(256, 8192),
            "train_steps": rng.randint(5, 40)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _lattice(key):
    """The workload's domain before any seed: built once, each state takes a copy."""
    c = dict(key)
    if c["kind"] == "channel":
        return scenarios.poiseuille(dx=c["dx"], H=c["H"], W=c["W"], scheme=c["scheme"])
    if c["kind"] == "dam2d":
        return scenarios.dam_break_2d(dx=c["dx"], L=c["L"], H=c["H"], TL=c["TL"], TH=c["TH"], scheme=c["scheme"])
    if c["closure"]:
        return les_case(c["dx"], L=c["L"], H=c["H"], W=c["W"], TL=c["TL"], TH=c["TH"], TW=c["W"])
    return scenarios.dam_break_3d(dx=c["dx"], L=c["L"], H=c["H"], W=c["W"], TL=c["TL"], TH=c["TH"], TW=c["W"])


def _smooth(x, L, rng, dim):
    """A smooth velocity field: a few Fourier modes of the extents L."""
    out = np.zeros((len(x), 3))
    for d in range(dim):
        for _ in range(2):
            k = rng.integers(1, 3, size=dim) * math.pi / L[:dim]
            out[:, d] += rng.uniform(-0.5, 0.5) * np.sin(x[:, :dim] @ k + rng.uniform(0.0, 2.0 * math.pi))
    return out


def _flow(case, seed):
    """(domain, dt, particles) of a fluid case: the lattice disordered by the seed."""
    dom, dt, info = _lattice(tuple(sorted((k, v) for k, v in case.items()
                                          if k not in ("name", "steps", "precision", "skin"))))
    rng = np.random.default_rng(seed)
    p = dom.particles.copy()
    x, free = p.get("x"), p.get("is_free") != 0
    dim, dx = dom.Dimension, case["dx"]
    U = 0.5 * info["umax"] if case["kind"] == "channel" else math.sqrt(9.81 * case["H"])
    nf = int(free.sum())
    xf = x[free]
    lo, hi = xf.min(0), xf.max(0)
    v = np.zeros_like(x)
    vf = U * _smooth(xf - lo, np.maximum(hi - lo, dx), rng, dim)
    vf[:, :dim] += 0.002 * U * (rng.random((nf, dim), dtype=np.float32) - 0.5)
    v[free] = vf
    xf[:, :dim] += 0.04 * dx * (rng.random((nf, dim), dtype=np.float32) - 0.5)
    x[free] = xf
    rho = p.get("density")
    rho[free] *= 1.0 + 2e-5 * (rng.random(nf, dtype=np.float32) - 0.5)
    p.set("x", x)
    p.set("v", v)
    p.set("density", rho)
    p.set("densityb", rho)
    return dom, dt, p


def _column_specs(case):
    n = case["n"]
    for q in range(n):
        t = (q + 0.5) / n
        yield (case["aspect0"] + (case["aspect1"] - case["aspect0"]) * t, 20.0 + 20.0 * ((q * 7) % n + 0.5) / n)


def _columns(case, seed):
    """[(domain, dt)] of a granular case: columns spread over the ensemble's aspect
    ratios and friction angles, each with noise in position, velocity and stress. The soil
    has the tests' 1 kPa cohesion: without it a free surface sits on the yield surface's
    apex, where the last bit of a stress decides the return mapping's branch."""
    rng = np.random.default_rng(seed)
    out = []
    for aspect, phi in _column_specs(case):
        dom, dt, info = scenarios.granular_column(dx=case["dx"], W=0.2, aspect=aspect, phi_deg=phi,
                                                     cohesion=1.0e3)
        p = dom.particles
        x, free = p.get("x"), p.get("is_free") != 0
        nf = int(free.sum())
        xf = x[free]
        v = np.zeros_like(x)
        v[free] = 0.05 * _smooth(xf - xf.min(0), np.array([0.2, info["H"], 1.0]), rng, 2)
        v[free, :2] += 0.002 * (rng.random((nf, 2)) - 0.5)
        x[free, :2] += 0.05 * case["dx"] * (rng.random((nf, 2)) - 0.5)
        sig = p.get("sigma")
        s = rng.uniform(-60.0, 60.0, size=(nf, 3))
        fi = np.flatnonzero(free)
        sig[fi, 0, 0] += s[:, 0]
        sig[fi, 1, 1] += s[:, 1]
        sig[fi, 0, 1] += s[:, 2]
        sig[fi, 1, 0] += s[:, 2]
        p.set("x", x)
        p.set("v", v)
        p.set("sigma", sig)
        out.append((dom, dt))
    return out


def _samples(case, seed):
    """Features like those of a coarse dam break, and coefficients that depend on them."""
    rng = np.random.default_rng(seed)
    n = case["samples"]
    f = np.empty((n, 6), np.float32)
    f[:, 0] = rng.normal(-6.0, 1.2, n)
    f[:, 1] = rng.normal(0.0, 0.08, n)
    f[:, 2] = f[:, 0] + rng.normal(0.3, 0.6, n)
    f[:, 3] = 1.0 + rng.normal(0.0, 3e-3, n)
    f[:, 4] = rng.choice([1.2, 1.3], n)
    f[:, 5] = rng.integers(20, 90, n)
    y = (0.05 + 0.04 * np.tanh(f[:, 0] + 6.0) + 0.3 * f[:, 1] ** 2 + 0.01 * rng.random(n)).astype(np.float32)
    return f, y


FLOW_FIELDS = ("x", "v", "density", "a", "ddensity")
SOIL_FIELDS = ("x", "v", "density", "a", "ddensity", "sigma")


def prepare(case, seed):
    if case["kind"] == "net":
        x, y = _samples(case, seed)
        net = ClosureNet(seed % 1000)
        net.set_data(x, y)
        return {"kind": "net", "net": net, "x": x, "case": case}
    if case["kind"] == "columns":
        cols = _columns(case, seed)
        cfgs = [dom.config(dt) for dom, dt in cols]
        for c in cfgs:
            c.precision = case["precision"]
        if case["n"] > 1:
            g = GpuEnsemble(cfgs)
            g.upload([dom.particles for dom, _ in cols])
        else:
            g = GpuDomain(cfgs[0])
            g.upload(cols[0][0].particles)
        return {"kind": "columns", "gpu": g, "case": case}
    dom, dt, p = _flow(case, seed)
    cfg = dom.config(dt)
    cfg.precision = case["precision"]
    g = GpuDomain(cfg)
    g.upload(p)
    st = {"kind": "flow", "gpu": g, "case": case}
    if case.get("closure"):
        st["net"] = ClosureNet.load(default_network_path())
        g.attach_closure(st["net"], case["dx"])
    if case.get("skin"):
        g.set_tuning(128, 1, 0, case["skin"])
    return st


def _typed(fields, case):
    if case["precision"] == FP64:
        return fields
    return {k: a if k == "x" else torch.from_numpy(a).to(torch.float32) for k, a in fields.items()}


def run(state):
    case = state["case"]
    if state["kind"] == "net":
        net = state["net"]
        losses = net.train(case["train_steps"], batch=case["batch"], lr=1e-3, seed=1)
        c = net.infer(state["x"])
        params, norm = net.get()
        return {"losses": losses, "c": c, "params": params, "norm": norm}
    g = state["gpu"]
    if state["kind"] == "columns":
        g.step(case["steps"])
        if case["n"] > 1:
            return [_typed(g.download_fields(q, SOIL_FIELDS), case) for q in range(case["n"])]
        return _typed(g.download_fields(SOIL_FIELDS), case)
    g.step(case["steps"])
    return _typed(g.download_fields(FLOW_FIELDS), case)


# ---------------------------------------------------------------------------
# work: what a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(case):
    """(free particles, all particles, in-support pairs with a free particle) of a case, from its lattice."""
    dx = case["dx"]
    if case["kind"] == "columns":
        free = allp = 0
        for aspect, _ in _column_specs(case):
            nf = round(0.2 / dx) * round(0.2 * aspect / dx)
            free += nf
            allp += nf + 3 * (round(0.2 * aspect / dx) + round(0.2 * (5.0 + aspect) / dx))
        return free, allp, free * math.pi * 2.4 ** 2 / 2.0
    if case["kind"] == "channel":
        nx, ny = round(case["W"] / dx), round(case["H"] / dx)
        return nx * ny, nx * (ny + 6), nx * ny * math.pi * 3.9 ** 2 / 2.0
    nx, ny = round(case["L"] / dx), round(case["H"] / dx)
    if case["kind"] == "dam2d":
        free = nx * ny
        return free, free + 3 * (round(case["TL"] / dx) + 6 + 2 * round(case["TH"] / dx)), free * math.pi * 2.4 ** 2 / 2.0
    nz = round(case["W"] / dx)
    tx, ty = round(case["TL"] / dx), round(case["TH"] / dx)
    free = nx * ny * nz
    walls = (tx + 6) * (ty + 3) * (nz + 6) - tx * ty * nz
    return free, free + walls, free * 4.0 / 3.0 * math.pi * 2.6 ** 3 / 2.0


def work(case):
    """Per step each particle's state (position, velocity, density, pressure and their
    history: 12 doubles; soil 4 stress and strain tensors more) is read and written once and
    each pair's force is evaluated once; then the fields are read back. A network sample takes
    a forward pass (17.3 kflop) and, in training, a backward pass of twice that."""
    if case["kind"] == "net":
        s, b = case["samples"], case["batch"] * case["train_steps"]
        return {"bytes": 28.0 * s + 28.0 * b + 3.0 * 4 * 8833 * case["train_steps"], "flops": 17.3e3 * s + 52.0e3 * b}
    free, allp, pairs = _counts(case)
    soil = case["kind"] == "columns"
    state = 2 * 8 * 12 * allp + (2 * 8 * 4 * 6 * free if soil else 0)
    back = 8 * (11 + (9 if soil else 0)) * allp
    return {"bytes": float(case["steps"] * state + back), "flops": float(case["steps"] * pairs * (180 if soil else 106))}


# ---------------------------------------------------------------------------
# exact: the same steps in plain torch, all in 64 bits
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _near(x, dim, reach, period):
    """Ordered pairs (i, j, x_i - x_j, r) of particles closer than reach, by a cell list."""
    lo, hi = x.min(0).values, x.max(0).values
    n, size = [1, 1, 1], [1.0, 1.0, 1.0]
    for d in range(dim):
        L = period[d] if period[d] > 0 else float(hi[d] - lo[d]) + 1e-9
        n[d] = max(1, int(L / (reach * (1 + 1e-9))))
        size[d] = L / n[d]
    cell = torch.zeros((len(x), 3), dtype=torch.int64, device=x.device)
    for d in range(dim):
        c = torch.floor((x[:, d] - lo[d]) / size[d]).to(torch.int64)
        cell[:, d] = c.remainder(n[d]) if period[d] > 0 else c.clamp(0, n[d] - 1)
    key = (cell[:, 2] * n[1] + cell[:, 1]) * n[0] + cell[:, 0]
    order = torch.argsort(key, stable=True)
    start = torch.zeros(n[0] * n[1] * n[2] + 1, dtype=torch.int64, device=x.device)
    start[1:] = torch.cumsum(torch.bincount(key, minlength=n[0] * n[1] * n[2]), 0)
    xs, cs = x[order], cell[order]
    I, J, D, R = [], [], [], []
    span = [(-1, 0, 1) if d < dim else (0,) for d in range(3)]
    for oz in span[2]:
        for oy in span[1]:
            for ox in span[0]:
                c = cs + torch.tensor([ox, oy, oz], device=x.device)
                ok = torch.ones(len(x), dtype=torch.bool, device=x.device)
                for d in range(dim):
                    if period[d] > 0:
                        c[:, d] = c[:, d].remainder(n[d])
                    else:
                        ok &= (c[:, d] >= 0) & (c[:, d] < n[d])
                k = torch.where(ok, (c[:, 2] * n[1] + c[:, 1]) * n[0] + c[:, 0], 0)
                b = start[k]
                cnt = torch.where(ok, start[k + 1] - b, 0)
                i = torch.repeat_interleave(torch.arange(len(x), device=x.device), cnt)
                first = torch.cumsum(cnt, 0) - cnt
                j = torch.arange(len(i), device=x.device) - first[i] + b[i]
                dxv = xs[i] - xs[j]
                for d in range(dim):
                    if period[d] > 0:
                        dxv[:, d] -= period[d] * torch.round(dxv[:, d] / period[d])
                r = dxv.square().sum(1).sqrt()
                keep = (r <= reach) & (i != j)
                I.append(order[i[keep]])
                J.append(order[j[keep]])
                D.append(dxv[keep])
                R.append(r[keep])
    return torch.cat(I), torch.cat(J), torch.cat(D), torch.cat(R)


def _kernel(kt, dim, q, h):
    """(W, (dW/dr) / r) of the cubic spline (0), Wendland (1) and quintic spline (2) kernels."""
    w = {0: (10 / (7 * math.pi), 1 / math.pi), 1: (7 / (4 * math.pi), 7 / (8 * math.pi)),
         2: (7 / (478 * math.pi), 1 / (120 * math.pi))}[kt][dim - 2] / h ** dim
    g = w / (h * h)
    z = torch.zeros_like(q)
    iq = 1.0 / torch.where(q > 0, q, 1.0)
    if kt == 0:
        W = torch.where(q < 1, 1 - 1.5 * q ** 2 + 0.75 * q ** 3, 0.25 * (2 - q).clamp(min=0) ** 3)
        G = torch.where(q < 1, -3 + 2.25 * q, -0.75 * (2 - q).clamp(min=0) ** 2 * iq)
    elif kt == 1:
        t = (1 - 0.5 * q).clamp(min=0)
        W, G = t ** 4 * (2 * q + 1), -5 * t ** 3
    else:
        a, b, c = (3 - q).clamp(min=0), (2 - q).clamp(min=0), (1 - q).clamp(min=0)
        W = a ** 5 - 6 * b ** 5 + 15 * c ** 5
        G = torch.where(q > 0, iq * (-5 * a ** 4 + 30 * b ** 4 - 75 * c ** 4), z - 120.0)
    return w * W, g * G


def _grid(dom, x, h, cellfac):
    """Lower corner and cell sizes of the reference's grid (they orient the wall pressure)."""
    lo, n, size = [], [], []
    for d in range(dom.Dimension):
        b, t = float(x[:, d].min()), float(x[:, d].max())
        pad = dom.R if dom.BC.Periodic[d] else h / 2
        b, t = b - pad, t + pad
        r = (t - b) / (cellfac * h)
        k = math.ceil(r) if math.ceil(r) - r < h / 10.0 else math.floor(r)
        lo.append(b)
        n.append(k)
        size.append((t - b) / k)
    return lo, n, size


def _sum(n, i, val):
    out = torch.zeros((n,) + val.shape[1:], dtype=torch.float64, device=val.device)
    return out.index_add_(0, i, val)


def _next_dt(dt, dti, bound):
    m = min(dti, bound)
    if dti > m:
        return 2 * dt * m / (dt + m) if dt < m else m
    return 2 * dt * dti / (dt + dti) if dti != dt else dti


def _fluid(dom, p, dt0, case):
    """Fields after the case's steps of a fluid domain."""
    dev, dim = _device(), dom.Dimension
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    kt = dom._kernel_type
    cellfac = 3.0 if kt == 2 else 2.0
    x, v, rho = T(p.get("x")), T(p.get("v")), T(p.get("density"))
    n = len(x)
    free = torch.as_tensor(p.get("is_free") != 0, device=dev)
    one = {k: float(p.get(k)[p.get("is_free") != 0][0]) for k in ("h", "cs", "alpha", "mass", "ref_density")}
    h, cs, alpha, m, rho0 = (one[k] for k in ("h", "cs", "alpha", "mass", "ref_density"))
    mass = T(p.get("mass"))
    eq = int(p.get("pres_eq")[0])
    mu_ref = float(p.get("mu_ref")[0])
    mu = T(p.get("mu"))
    les = bool(case.get("closure"))
    grav = torch.tensor(dom.Gravity, dtype=torch.float64, device=dev)
    body = torch.tensor(dom.BodyForce, dtype=torch.float64, device=dev)
    oriented = bool((grav != 0).any())
    lo, ncell, size = _grid(dom, p.get("x"), h, cellfac)
    period = [0.0, 0.0, 0.0]
    top = list(lo)
    for d in range(dim):
        top[d] = lo[d] + ncell[d] * size[d]
        if dom.BC.Periodic[d]:
            period[d] = top[d] - lo[d]

    def eos(r):
        return cs * cs * (r - rho0) if eq == 0 else rho0 * cs * cs / 7.0 * ((r / rho0) ** 7 - 1)

    def inverse(pr):
        return pr / (cs * cs) + rho0 if eq == 0 else (pr * 7.0 / (rho0 * cs * cs) + 1) ** (1 / 7) * rho0

    def sound(r):
        return torch.full_like(r, cs) if eq == 0 else cs * (r / rho0) ** 3

    net = np.load(default_network_path()) if les else None
    pr = eos(rho)
    hist_v, hist_r = torch.zeros_like(v), torch.zeros_like(rho)
    dt, dti, ct, first = dt0, dt0, 30, True
    for _ in range(case["steps"]):
        i, j, d, r = _near(x, dim, cellfac * h, period)
        K, G = _kernel(kt, dim, r / h, h)
        # walls: pressure and velocity of their free neighbours
        w = ~free[i] & free[j]
        wi, wj, wk = i[w], j[w], K[w]
        sk = _sum(n, wi, wk)
        gd = d[w] @ grav
        if oriented:
            c = torch.stack([torch.floor((x[:, k] - lo[k]) / size[k]).clamp(0, ncell[k] - 1) for k in range(dim)], 1)
            o = c[wj] - c[wi]
            sign = torch.where(wi > wj, 1.0, -1.0).to(torch.float64)
            for k in range(dim):
                sign = torch.where(o[:, k] != 0, torch.sign(o[:, k]), sign)
            gd = gd * sign
        has = sk > 0
        safe = torch.where(has, sk, 1.0)
        pw = torch.where(has, _sum(n, wi, pr[wj] * wk + gd * rho[wj] * wk) / safe, 0.0)
        nsv = torch.where(has[:, None], _sum(n, wi, v[wj] * wk[:, None]) / safe[:, None], 0.0)
        pr = torch.where(free, pr, pw)
        seen = torch.where(free, rho, inverse(pw))
        snd = sound(seen)
        # pair forces on the free particles
        f = free[i]
        i, j, d, r, K, G = i[f], j[f], d[f], r[f], K[f], G[f]
        fj = free[j]
        mj = torch.where(fj, mass[j], mass[i])
        dv = v[i] - v[j]
        vx = (dv * d).sum(1)
        D = r * r + 0.01 * h * h
        PI = torch.where(vx < 0, -alpha * 0.5 * (snd[i] + snd[j]) * h * vx / D / (0.5 * (seen[i] + seen[j])), 0.0)
        vab = torch.where(fj[:, None], dv, v[i] - (2 * v[j] - nsv[j]))
        if les:
            Mu = torch.where(fj, 2 * mu[i] * mu[j] / (mu[i] + mu[j]), mu[i])
        else:
            Mu = mu[i]
        s = -(pr[i] / seen[i] ** 2 + pr[j] / seen[j] ** 2 + PI) * G
        acc = mj[:, None] * (s[:, None] * d + (2 * Mu / (seen[i] * seen[j]) * G)[:, None] * vab)
        a = grav + _sum(n, i, acc) + body * free[:, None]
        dr = _sum(n, i, mj * seen[i] / seen[j] * G * vx)
        if dim == 2:
            a[:, 2] = torch.where(free, 0.0, a[:, 2])
        if les:
            c2 = -G * mj / seen[j]
            M = _sum(n, i, c2[:, None, None] * vab[:, :, None] * d[:, None, :])
            S, A = M + M.mT, M - M.mT
            tmp = S.square().sum((1, 2))
            shear = (0.5 * tmp).sqrt()
            vort = (0.5 * A.square().sum((1, 2))).sqrt()
            nnb = torch.bincount(i, minlength=n).to(torch.float64)
            r3 = torch.where(tmp > 0, torch.linalg.det(S) / torch.where(tmp > 0, tmp, 1.0) ** 1.5, 0.0)
            c = _coefficient(net, torch.stack([torch.log((shear * h / cs).clamp(min=1e-12)), r3,
                                               torch.log((vort * h / cs).clamp(min=1e-12)), rho / rho0,
                                               torch.full_like(rho, h / case["dx"]), nnb], 1))
            nut = torch.where(c >= 0, c * h * h * shear, (0.17 * h) ** 2 * 2 * shear)
            mu = torch.where(free, mu_ref + rho0 * nut, mu)
        an = a[free].norm(dim=1).max()
        dt = _next_dt(dt, dti, float(dom.sqrt_h_a * torch.sqrt(h / an)))
        fr = free[:, None]
        if dom.Scheme == 0:
            x = torch.where(fr, x + dt * v + 0.5 * dt * dt * a, x)
            ov, orho = v, rho
            if ct == 30:
                v, rho = torch.where(fr, v + dt * a, v), torch.where(free, rho + dt * dr, rho)
            else:
                v, rho = torch.where(fr, hist_v + 2 * dt * a, v), torch.where(free, hist_r + 2 * dt * dr, rho)
            hist_v, hist_r = ov, orho
            ct = 0 if ct == 30 else ct + 1
        else:
            if first:
                hist_v, hist_r = v - dt / 2 * a, rho - dt / 2 * dr
            nv, nr = hist_v + dt * a, hist_r + dt * dr
            v, rho = torch.where(fr, (nv + hist_v) / 2, v), torch.where(free, (nr + hist_r) / 2, rho)
            x = torch.where(fr, x + dt * nv, x)
            hist_v, hist_r = nv, nr
        first = False
        for k in range(dim):
            if period[k] > 0:
                x[:, k] = torch.where(x[:, k] > top[k], x[:, k] - period[k], x[:, k])
                x[:, k] = torch.where(x[:, k] < lo[k], x[:, k] + period[k], x[:, k])
        pr = torch.where(free, eos(rho), pr)
    dr = torch.where(free, dr, 0.0)
    return {"x": x, "v": v, "density": rho, "a": a, "ddensity": dr}


def _coefficient(net, feat):
    """The network's coefficient, or -1 outside its training range (rates below it are raised to its floor)."""
    dev = feat.device
    q = torch.as_tensor(net["params"].astype(np.float32), device=dev)
    nrm = torch.as_tensor(net["norm"], dtype=torch.float64, device=dev)
    mean, inv, low, high = nrm[0:6], nrm[6:12], nrm[12:18], nrm[18:24]
    feat = feat.clone()
    for k in (0, 2):
        feat[:, k] = feat[:, k].clamp(min=float(low[k]))
    seen = feat.to(torch.float32).to(torch.float64)  # the range is kept in FP32: h / dx lies on its edge
    inside = ((seen >= low) & (seen <= high)).all(1)
    at, sizes = 0, [(64, 6), (64,), (64, 64), (64,), (64, 64), (64,), (64,), (1,)]
    W = []
    for s in sizes:
        k = int(np.prod(s))
        t = q[at:at + k].reshape(s)
        W.append((t.to(torch.bfloat16) if len(s) == 2 else t).to(torch.float64))
        at += k
    z = (feat - mean) * inv
    for k in (0, 2, 4):
        z = torch.nn.functional.silu(z @ W[k].T + W[k + 1])
    return torch.where(inside, torch.nn.functional.softplus(z @ W[6] + W[7]), -1.0)


def _tensile(S, ti, rho):
    """The tensile-instability stress of 2D stresses S (n, 3, 3): minus ti / rho^2 of the tensile principal stresses."""
    half, shear = 0.5 * (S[:, 0, 0] - S[:, 1, 1]), S[:, 0, 1]
    mean, rad = 0.5 * (S[:, 0, 0] + S[:, 1, 1]), torch.hypot(half, shear)
    e = [torch.where(p > 0, -ti * p / (rho * rho), 0.0) for p in (mean + rad, mean - rad)]
    c, s = (t / torch.where(rad > 0, rad, 1.0) for t in (half, shear))  # cosine and sine of twice the angle
    m, r = 0.5 * (e[0] + e[1]), 0.5 * (e[0] - e[1])
    out = torch.zeros_like(S)
    out[:, 0, 0], out[:, 1, 1] = m + r * c, m - r * c
    out[:, 0, 1] = out[:, 1, 0] = r * s
    return out


def _soil(dom, dt0, case):
    """Fields after the case's steps of a 2D Drucker-Prager column (Modified Verlet)."""
    dev, p = _device(), dom.particles
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    x, v, rho, mass, sig = (T(p.get(k)) for k in ("x", "v", "density", "mass", "sigma"))
    n = len(x)
    free = torch.as_tensor(p.get("is_free") != 0, device=dev)
    h, cs, al, be, ti, tin, tid, G_, K_, phi, coh = (
        float(p.get(k)[0])
        for k in ("h", "cs", "alpha", "beta", "ti", "tin", "ti_init_dist", "g_mod", "k_mod", "phi", "cohesion"))
    tan = math.tan(phi)
    da, kf = (c / math.sqrt(9 + 12 * tan * tan) for c in (tan, 3 * coh))  # Drucker-Prager, plane strain
    grav = torch.tensor(dom.Gravity, dtype=torch.float64, device=dev)
    eye = torch.eye(3, dtype=torch.float64, device=dev)
    eye2 = torch.diag(torch.tensor([1.0, 1.0, 0.0], dtype=torch.float64, device=dev))
    tir = torch.zeros_like(sig)
    Wd = _kernel(0, 2, torch.tensor([tid / h], dtype=torch.float64, device=dev), h)[0]
    hv, hr, hs = torch.zeros_like(v), torch.zeros_like(rho), torch.zeros_like(sig)
    dt, dti, ct = dt0, dt0, 30

    def tr(t):
        return t[:, 0, 0] + t[:, 1, 1] + t[:, 2, 2]

    def apex(S):
        I1 = tr(S)
        return torch.where((da * I1 > kf)[:, None, None], S - ((I1 - kf / da) / 3)[:, None, None] * eye, S)

    def dev_of(S):
        D = S - (tr(S) / 3)[:, None, None] * eye
        return D, 0.5 * (D * D.mT).sum((1, 2))

    for _ in range(case["steps"]):
        i, j, d, r = _near(x, 2, 2 * h, [0.0] * 3)
        K, G = _kernel(0, 2, r / h, h)
        w = ~free[i] & free[j]
        wi, wj, wk = i[w], j[w], K[w]
        sk = _sum(n, wi, wk)
        has = sk > 0
        safe = torch.where(has, sk, 1.0)
        ws = torch.where(has[:, None, None], _sum(n, wi, sig[wj] * wk[:, None, None]) / safe[:, None, None], 0.0)
        ns = torch.where(has[:, None], _sum(n, wi, v[wj] * wk[:, None]) / safe[:, None], 0.0)
        sig = torch.where(free[:, None, None], sig, ws)
        tir = torch.where((free | has)[:, None, None], _tensile(sig, ti, rho), tir)
        f = free[i]
        i, j, d, r, K, G = i[f], j[f], d[f], r[f], K[f], G[f]
        fj = free[j]
        mj = torch.where(fj, mass[j], mass[i])
        dj = torch.where(fj, rho[j], rho[i])
        di = rho[i]
        dv = v[i] - v[j]
        vx = (dv * d).sum(1)
        D = r * r + 0.01 * h * h
        t = h * vx
        PI = torch.where(vx < 0, t * (al * cs * D + be * t) / (D * D * 0.5 * (di + dj)), 0.0)
        vab = torch.where(fj[:, None], dv, v[i] - (2 * v[j] - ns[j]))
        M = sig[i] / (di * di)[:, None, None] + sig[j] / (dj * dj)[:, None, None] + PI[:, None, None] * eye2
        M = M + (tir[i] + tir[j]) * ((K / Wd) ** tin)[:, None, None]
        g = G[:, None] * d
        a = grav + _sum(n, i, mj[:, None] * torch.einsum("nr,nrc->nc", g, M))
        a[:, 2] = torch.where(free, 0.0, a[:, 2])
        dr = _sum(n, i, mj * di / dj * (dv * g).sum(1))
        B = _sum(n, i, (-0.5 * G * mj / dj)[:, None, None] * vab[:, :, None] * d[:, None, :])
        S, R = B + B.mT, B - B.mT
        an = a[free].norm(dim=1).max()
        dt = _next_dt(dt, dti, float(dom.sqrt_h_a * torch.sqrt(h / an)))
        fr = free[:, None]
        x = torch.where(fr, x + dt * v + 0.5 * dt * dt * a, x)
        ov, orho, osig = v, rho, sig
        I1s = tr(S)
        X = (I1s * K_)[:, None, None] * eye + 2 * G_ * (S - (I1s / 3)[:, None, None] * eye) + sig @ R.mT + R @ sig
        fac = dt if ct == 30 else 2 * dt
        base_v, base_r, base_s = (v, rho, sig) if ct == 30 else (hv, hr, hs)
        v = torch.where(fr, base_v + fac * a, v)
        rho = torch.where(free, base_r + fac * dr, rho)
        new = apex(base_s + fac * X)
        Dn, J2 = dev_of(new)
        plastic = J2.sqrt() + da * tr(new) > kf
        Do, J2o = dev_of(osig)
        q = J2o.sqrt()
        act = plastic & (q > 0)
        qs = torch.where(q > 0, q, 1.0)
        dL = (3 * da * K_ * I1s + G_ / qs * (Do * S).sum((1, 2))) / (9 * da * da * K_ + G_)
        flow = (3 * da * K_) * eye2 + Do * (G_ / qs)[:, None, None]
        new = torch.where(act[:, None, None], new - flow * (dL * fac)[:, None, None], new)
        new = torch.where(plastic[:, None, None], apex(new), new)
        Dn, J2 = dev_of(new)
        q, I1 = J2.sqrt(), tr(new)
        over = plastic & (q + da * I1 > kf) & (q > 0)
        back = (I1 / 3)[:, None, None] * eye + Dn * ((kf - da * I1) / torch.where(q > 0, q, 1.0))[:, None, None]
        new = torch.where(over[:, None, None], back, new)
        sig = torch.where(free[:, None, None], new, sig)
        hv, hr, hs = ov, orho, osig
        ct = 0 if ct == 30 else ct + 1
    return {"x": x, "v": v, "density": rho, "a": a, "ddensity": torch.where(free, dr, 0.0), "sigma": sig}


def exact(case, seed):
    if case["kind"] == "net":
        return None  # Adam's path from FP32 and BF16 arithmetic: no 64-bit values to hold it to
    if case["kind"] == "columns":
        got = [{k: t.cpu() for k, t in _soil(dom, dt, case).items()} for dom, dt in _columns(case, seed)]
        return got if case["n"] > 1 else got[0]
    free, _, pairs = _counts(case)
    if pairs * case["steps"] > 2.5e9 or (pairs > 1e8):
        return None  # over 20 seconds
    dom, dt, p = _flow(case, seed)
    return {k: t.cpu() for k, t in _fluid(dom, p, dt, case).items()}
