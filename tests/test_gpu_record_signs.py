"""Negative densities in the FP32C pair kernels: what kind a neighbour is never
follows from the sign of its density. Walls under strong suction (the inverse
EOS with PresEq 0 gives them a negative density) and free particles with one,
one step from that state against the oracle, at the form's parity bound: 1e-5 of
each particle's sum of term magnitudes."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain
from tests.gpu_helpers import oracle_state

pytestmark = pytest.mark.gpu


def check(dom, dt, change, rates=()):
    cfg = dom.config(dt)
    o = OracleDomain(cfg, dom.particles, initial=True)
    state = oracle_state(o)
    change(state)
    grid, integ = o.grid(), o.integrator()
    o = OracleDomain(cfg, state, initial=False, grid=grid, integ=integ)
    cfg.precision = 1
    gd = GpuDomain(cfg, grid=grid, integ=integ)
    gd.upload(state, initial=False)
    o.step(1)
    gd.step(1)
    a_scale, dr_scale = o.scales()
    ref, got = o.download(), gd.download_fields()
    f = ref["is_free"] == 1
    assert np.max(np.linalg.norm(got["a"] - ref["a"], axis=1)[f] / a_scale[f]) <= 1e-5
    assert np.max(np.abs(got["ddensity"] - ref["ddensity"])[f] / (dr_scale[f] + 1e-300)) <= 1e-5
    for k in rates:
        assert np.max(np.abs(got[k] - ref[k])[f]) <= 1e-5 * np.abs(ref[k][f]).max(), k
    gd.close()


def stirred(dom, dx, dim):
    rng = np.random.default_rng(5)
    p = dom.particles
    free = p.get("is_free") != 0
    x, v = p.get("x"), p.get("v")
    x[free, :dim] += 0.1 * dx * (rng.random((int(free.sum()), dim)) - 0.5)
    v[free, :dim] += 0.5 * (rng.random((int(free.sum()), dim)) - 0.5)
    p.set("x", x)
    p.set("v", v)


def tank(dim):
    if dim == 2:
        dx = 0.031
        dom, dt, info = scenarios.dam_break_2d(dx=dx, L=0.4, H=0.7, TL=1.1, TH=0.9)
    else:
        dx = 0.05
        dom, dt, info = scenarios.dam_break_3d(dx=dx, L=0.3, H=0.45, W=0.25, TL=0.6, TH=0.5, TW=0.25)
    stirred(dom, dx, dim)
    return dom, dt, info


@pytest.mark.parametrize("slip", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_walls_under_suction(gpu, dim, slip):
    dom, dt, info = tank(dim)
    p = dom.particles
    p.set("pres_eq", 0)
    if slip:
        p.set("no_slip", 0)

    def change(s):
        near = (s.get("is_free") != 0) & (s.get("x")[:, 1] < 0.1) & (s.get("x")[:, 0] > 0.1)
        pr = s.get("pressure")
        pr[near] = -3.0 * info["cs"] ** 2 * 1000.0
        s.set("pressure", pr)

    check(dom, dt, change)


@pytest.mark.parametrize("eos", [0, 1])
@pytest.mark.parametrize("dim", [2, 3])
def test_negative_free_density(gpu, dim, eos):
    dom, dt, info = tank(dim)
    dom.particles.set("pres_eq", eos)

    def change(s):
        x = s.get("x")
        inner = np.flatnonzero((s.get("is_free") != 0) & (x[:, 1] > 0.15) & (x[:, 0] > 0.12))
        d = s.get("density")
        d[inner[::7]] *= -0.5
        s.set("density", d)

    check(dom, dt, change)


def test_negative_soil_density(gpu):
    dx = 0.013
    dom, dt, _ = scenarios.granular_column(dx=dx, aspect=0.8, cohesion=1.0e3)
    stirred(dom, dx, 2)

    def change(s):
        free = np.flatnonzero(s.get("is_free") != 0)
        d = s.get("density")
        d[free[::7]] *= -0.5
        s.set("density", d)

    check(dom, dt, change, ("strain_rate", "rotation_rate"))


def test_walls_out_of_reach(gpu):
    """A background pressure under which the inverse Tait equation has no value at
    p = 0: walls that stand in a list (one with a skin) but in no free particle's
    support leave its sums alone."""
    dom, dt, info = tank(2)
    p = dom.particles
    p.set("p0", 0.5 * 1000.0 * info["cs"] ** 2)
    x = p.get("x")
    x[p.get("is_free") == 0, 1] -= 0.3 * 0.031  # a floor just out of some supports
    p.set("x", x)
    cfg = dom.config(dt)
    o = OracleDomain(cfg, p, initial=True)
    o.step(1)
    ref = o.download()
    cfg.precision = 1
    for skin in (0, 150):
        gd = GpuDomain(cfg)
        gd.upload(p)
        gd.set_tuning(128, 1, 0, skin)
        gd.step(1)
        got = gd.download_fields()
        a_scale, _ = o.scales()
        f = ref["is_free"] == 1
        assert np.max(np.linalg.norm(got["a"] - ref["a"], axis=1)[f] / a_scale[f]) <= 1e-5
        gd.close()
