"""FP32C fluids whose classes share their pair constants but not their flags (a
slip lid over no-slip walls, LES or a yield stress on part of the fluid): one
step against the oracle at the form's parity bound, 1e-5 of each particle's sum
of term magnitudes, with short lists and with lists longer than their capacity."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,kernel,hfac", [(2, 0, 1.2), (2, 0, 3.2), (2, 2, 1.1), (3, 1, 1.3), (3, 1, 1.9),
                                             (3, 2, 1.0)])
@pytest.mark.parametrize("kind", ["lid", "les", "bingham"])
def test_unlike_flags(gpu, kind, dim, kernel, hfac):
    if dim == 2:
        dx = 0.031
        dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.4, H=0.7, TL=1.1, TH=0.9, kernel=kernel, hfac=hfac)
    else:
        dx = 0.05
        dom, dt, _ = scenarios.dam_break_3d(dx=dx, L=0.3, H=0.35, W=0.25, TL=0.6, TH=0.4, TW=0.25, kernel=kernel,
                                            hfac=hfac)
    p = dom.particles
    x = p.get("x")
    free = p.get("is_free") != 0
    rng = np.random.default_rng(11)
    v = p.get("v")
    x[free, :dim] += 0.1 * dx * (rng.random((int(free.sum()), dim)) - 0.5)
    v[free, :dim] += 0.5 * (rng.random((int(free.sum()), dim)) - 0.5)
    p.set("x", x)
    p.set("v", v)
    slip = p.get("no_slip")
    slip[~free & (x[:, 1] > 0.2)] = 0
    p.set("no_slip", slip)
    left = (x[:, 0] < 0.2).astype(np.int32)
    if kind == "les":
        p.set("les", left)
        p.set("csmag", 0.17)
    elif kind == "bingham":
        p.set("t0", 5.0 * left)
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
    if kind != "lid":
        s = np.abs(ref["strain_rate"][f]).max()
        assert np.max(np.abs(got["strain_rate"] - ref["strain_rate"])[f]) <= 1e-5 * s
    gd.close()
