"""Ensembles whose instances differ in the parameters that choose a pair kernel's
form or its constants (artificial viscosity, lattice, viscosity, wall masses,
equation of state, slip, soil moduli, tensile instability): each instance still
evolves bit for bit as the same domain alone, in both forms. (Instances with and
without LES or a yield stress agree to rounding only.)"""
import numpy as np
import pytest

from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain, GpuEnsemble

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "density", "pressure", "a", "ddensity", "sigma", "zwab")


def stirred(dom, dt, dx, params):
    rng = np.random.default_rng(3)
    p = dom.particles
    d = dom.Dimension
    free = p.get("is_free") != 0
    x, v = p.get("x"), p.get("v")
    x[free, :d] += 0.05 * dx * (rng.random((int(free.sum()), d)) - 0.5)
    v[free, :d] += 0.2 * (rng.random((int(free.sum()), d)) - 0.5)
    p.set("x", x)
    p.set("v", v)
    for k, a in params.items():
        if k == "lid":  # slip walls above a height: flags differ within the instance
            slip = p.get("no_slip")
            slip[~free & (p.get("x")[:, 1] > a)] = 0
            p.set("no_slip", slip)
        elif k == "right_cs":  # two equations of state within the instance
            cs = p.get("cs")
            cs[p.get("x")[:, 0] > 0.2] = a
            p.set("cs", cs)
        else:
            p.set(k, a)
    return dom, 0.2 * dt


def dam2(dx=0.04, kernel=0, **params):
    dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.4, H=0.6, TL=1.0, TH=0.8, kernel=kernel)
    return stirred(dom, dt, dx, params)


def dam3(dx=0.05, **params):
    dom, dt, _ = scenarios.dam_break_3d(dx=dx, L=0.3, H=0.35, W=0.25, TL=0.6, TH=0.4, TW=0.25)
    return stirred(dom, dt, dx, params)


def column(dx=0.02, E=0.84e6, **params):
    dom, dt, _ = scenarios.granular_column(dx=dx, aspect=0.8, cohesion=1.0e3, E=E)
    return stirred(dom, dt, dx, params)


CASES = {
    "alpha": lambda: [dam2(), dam2(alpha=0.3)],
    "alpha_beta": lambda: [dam2(alpha=0.0), dam2(alpha=0.1, beta=0.1)],
    "lattice": lambda: [dam2(), dam2(0.05)],
    "lattice_quintic": lambda: [dam2(kernel=2), dam2(0.05, kernel=2), dam2(alpha=0.2, kernel=2)],
    "lattice_3d": lambda: [dam3(), dam3(0.06)],
    "lattice_general": lambda: [dam3(lid=0.1), dam3(0.06, lid=0.1), dam3(ti=0.3, ti_init_dist=0.05)],
    "viscosity": lambda: [dam2(), dam2(mu=0.1, mu_ref=0.1)],
    "wall_mass": lambda: [dam2(), dam2(fpmassc=0.8)],
    "sound_speed": lambda: [dam2(), dam2(cs=60.0)],
    "state_equation": lambda: [dam2(), dam2(pres_eq=0)],
    "slip": lambda: [dam2(), dam2(no_slip=0)],
    "lid": lambda: [dam2(), dam2(lid=0.3)],  # one instance in each form
    "tension": lambda: [dam2(), dam2(ti=0.3, ti_init_dist=0.04), dam2(alpha=0.3)],
    "several_eos": lambda: [dam2(ti=0.3, ti_init_dist=0.04), dam2(right_cs=60.0), dam2(lid=0.3), dam2()],
    "soil_lattice": lambda: [column(), column(0.03)],
    "soil_modulus": lambda: [column(), column(E=1.5e6)],
    "soil_tension": lambda: [column(), column(ti=0.0), column(tin=3.0)],
    "soil_slip": lambda: [column(), column(no_slip=0), column(lid=0.1)],
    "soil_wall_mass": lambda: [column(), column(fpmassc=0.8)],
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", list(CASES))
def test_unlike_instances(gpu, name, precision):
    doms = CASES[name]()
    cfgs = []
    for dom, dt in doms:
        cfg = dom.config(dt)
        cfg.precision = precision
        cfgs.append(cfg)
    ens = GpuEnsemble(cfgs)
    ens.upload([dom.particles for dom, _ in doms])
    ens.step(4)
    for q, (dom, _) in enumerate(doms):
        gd = GpuDomain(cfgs[q])
        gd.upload(dom.particles)
        gd.step(4)
        ref, got = gd.download_fields(FIELDS), ens.download_fields(q, FIELDS)
        for f in FIELDS:
            np.testing.assert_array_equal(got[f], ref[f], err_msg=f"{name} instance {q} field {f}")
        gd.close()
    ens.close()
