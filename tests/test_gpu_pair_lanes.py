"""Pair kernels at the sizes and options where their lane groups and the
constant-parameter form can go wrong, one step against the oracle: particle
counts that leave groups, warps and blocks partly filled, lists longer than
their capacity (the cell scan), every kernel, beta and wall masses, free-slip
walls, and tensile stresses. The tolerances are the forms' parity bounds: 1e-12
(FP64) and 1e-5 (FP32C) of each particle's sum of term magnitudes."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain
from tests.gpu_helpers import assert_step_parity

pytestmark = pytest.mark.gpu


def one_step(dom, dt, label):
    cfg = dom.config(dt)
    o = OracleDomain(cfg, dom.particles, initial=True)
    o.step(1)
    gd = GpuDomain(cfg)
    gd.upload(dom.particles)
    gd.step(1)
    a_scale, dr_scale = o.scales()
    assert_step_parity(gd.download_fields(), o.download(), a_scale, dr_scale, dt, label=label)
    gd.close()


def stir(p, dx, seed, dim, speed):
    rng = np.random.default_rng(seed)
    free = p.get("is_free") != 0
    x, v = p.get("x"), p.get("v")
    x[free, :dim] += 0.1 * dx * (rng.random((int(free.sum()), dim)) - 0.5)
    v[free, :dim] += speed * (rng.random((int(free.sum()), dim)) - 0.5)
    p.set("x", x)
    p.set("v", v)


@pytest.mark.parametrize("dx", [0.05, 0.031])
@pytest.mark.parametrize("kernel,hfac,beta,fpmassc,slip", [
    (0, 1.2, 0.0, 1.0, False), (0, 2.7, 0.0, 1.0, False), (1, 1.3, 0.2, 1.0, False), (2, 1.1, 0.0, 0.8, False),
    (1, 1.2, 0.0, 1.0, True)])
def test_fluid_2d(gpu, dx, kernel, hfac, beta, fpmassc, slip):
    dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.4, H=0.7, TL=1.1, TH=0.9, kernel=kernel, hfac=hfac)
    p = dom.particles
    p.set("beta", beta)
    p.set("fpmassc", fpmassc)
    if slip:
        p.set("no_slip", 0)
    stir(p, dx, 3, 2, 0.5)
    one_step(dom, dt, f"2D kernel {kernel} hfac {hfac}")


@pytest.mark.parametrize("kernel,hfac", [(1, 1.3), (1, 1.7), (2, 1.1)])
def test_fluid_3d(gpu, kernel, hfac):
    dom, dt, _ = scenarios.dam_break_3d(dx=0.05, L=0.3, H=0.35, W=0.25, TL=0.6, TH=0.4, TW=0.25, kernel=kernel,
                                        hfac=hfac)
    stir(dom.particles, 0.05, 4, 3, 0.5)
    one_step(dom, dt, f"3D kernel {kernel} hfac {hfac}")


@pytest.mark.parametrize("hfac,ti,alpha", [(1.2, 0.5, 0.1), (2.7, 0.5, 0.1), (1.2, 0.0, 0.0)])
def test_soil_2d(gpu, hfac, ti, alpha):
    dx = 0.013
    dom, dt, info = scenarios.granular_column(dx=dx, aspect=0.8, cohesion=1.0e3, hfac=hfac, ti=ti, alpha=alpha)
    p = dom.particles
    stir(p, dx, 5, 2, 0.05)
    rng = np.random.default_rng(6)  # some particles in tension: both branches of the tensile-instability term
    free = np.flatnonzero(p.get("is_free") != 0)
    s = p.get("sigma")
    s[free, 0, 0] += rng.uniform(-400.0, 400.0, len(free))
    s[free, 1, 1] += rng.uniform(-400.0, 400.0, len(free))
    p.set("sigma", s)
    one_step(dom, dt, f"soil hfac {hfac} ti {ti}")


@pytest.mark.parametrize("les", [False, True])
@pytest.mark.parametrize("dim,kernel,hfac,beta,fpmassc,slip", [
    (2, 0, 1.2, 0.0, 1.0, False), (2, 0, 3.2, 0.2, 1.0, False), (2, 2, 1.1, 0.0, 0.8, False),
    (2, 1, 1.3, 0.1, 1.0, True), (3, 1, 1.3, 0.0, 1.0, False), (3, 1, 1.9, 0.2, 0.7, False),
    (3, 0, 1.3, 0.0, 1.0, True), (3, 2, 1.0, 0.0, 1.0, False)])
def test_fluid_fp32c(gpu, dim, kernel, hfac, beta, fpmassc, slip, les):
    if dim == 2:
        dx = 0.031
        dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.4, H=0.7, TL=1.1, TH=0.9, kernel=kernel, hfac=hfac)
    else:
        dx = 0.05
        dom, dt, _ = scenarios.dam_break_3d(dx=dx, L=0.3, H=0.35, W=0.25, TL=0.6, TH=0.4, TW=0.25, kernel=kernel,
                                            hfac=hfac)
    p = dom.particles
    p.set("beta", beta)
    p.set("fpmassc", fpmassc)
    if slip:
        p.set("no_slip", 0)
    if les:
        p.set("les", 1)
        p.set("csmag", 0.17)
    stir(p, dx, 7, dim, 0.5)
    o = OracleDomain(dom.config(dt), p, initial=True)
    o.step(1)
    a_scale, dr_scale = o.scales()
    ref = o.download()
    cfg = dom.config(dt)
    cfg.precision = 1
    gd = GpuDomain(cfg)
    gd.upload(p)
    gd.step(1)
    got = gd.download_fields()
    free = ref["is_free"] == 1
    assert np.max(np.linalg.norm(got["a"] - ref["a"], axis=1)[free] / a_scale[free]) <= 1e-5
    assert np.max(np.abs(got["ddensity"] - ref["ddensity"])[free] / (dr_scale[free] + 1e-300)) <= 1e-5
    if les:
        s = np.abs(ref["strain_rate"][free]).max()
        assert np.max(np.abs(got["strain_rate"] - ref["strain_rate"])[free]) <= 1e-5 * s
    gd.close()


@pytest.mark.parametrize("kernel", [0, 1, 2])
@pytest.mark.parametrize("hfac,ti,alpha,fpmassc,slip", [
    (1.2, 0.5, 0.1, 1.0, False), (3.2, 0.5, 0.1, 0.9, False), (1.2, 0.0, 0.0, 1.0, True)])
def test_soil_fp32c(gpu, kernel, hfac, ti, alpha, fpmassc, slip):
    dx = 0.013
    dom, dt, info = scenarios.granular_column(dx=dx, aspect=0.8, cohesion=1.0e3, hfac=hfac, ti=ti, alpha=alpha)
    dom.Kernel_Set(kernel)
    p = dom.particles
    p.set("fpmassc", fpmassc)
    if slip:
        p.set("no_slip", 0)
    stir(p, dx, 8, 2, 0.5)
    rng = np.random.default_rng(9)
    free = np.flatnonzero(p.get("is_free") != 0)
    s = p.get("sigma")
    for r, c in ((0, 0), (1, 1)):
        s[free, r, c] += rng.uniform(-400.0, 400.0, len(free))
    p.set("sigma", s)
    o = OracleDomain(dom.config(dt), p, initial=True)
    o.step(1)
    a_scale, dr_scale = o.scales()
    ref = o.download()
    cfg = dom.config(dt)
    cfg.precision = 1
    gd = GpuDomain(cfg)
    gd.upload(p)
    gd.step(1)
    got = gd.download_fields()
    f = ref["is_free"] == 1
    assert np.max(np.linalg.norm(got["a"] - ref["a"], axis=1)[f] / a_scale[f]) <= 1e-5
    assert np.max(np.abs(got["ddensity"] - ref["ddensity"])[f] / (dr_scale[f] + 1e-300)) <= 1e-5
    for k in ("strain_rate", "rotation_rate", "sigma", "strain"):
        assert np.max(np.abs(got[k] - ref[k])[f]) <= 1e-5 * np.abs(ref[k][f]).max(), k
    gd.close()
