"""A fluid whose particles have unlike equations of state: a wall takes its density
from its partner's, pair by pair, in the FP32C form as in FP64. One step against
the oracle at the forms' parity bounds."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("what,value", [("cs", 60.0), ("pres_eq", 0), ("ref_density", 990.0), ("pres_eq", 2)])
@pytest.mark.parametrize("dim", [2, 3])
def test_two_equations_of_state(gpu, dim, what, value, precision):
    if dim == 2:
        dom, dt, _ = scenarios.dam_break_2d(dx=0.04, L=0.4, H=0.6, TL=1.0, TH=0.8)
    else:
        dom, dt, _ = scenarios.dam_break_3d(dx=0.05, L=0.3, H=0.35, W=0.25, TL=0.6, TH=0.4, TW=0.25)
    dt *= 0.2
    p = dom.particles
    a = p.get(what)
    a[p.get("x")[:, 0] > 0.2] = value
    p.set(what, a)
    rng = np.random.default_rng(1)
    free = p.get("is_free") != 0
    v = p.get("v")
    v[free, :dim] += 0.5 * (rng.random((int(free.sum()), dim)) - 0.5)
    p.set("v", v)
    o = OracleDomain(dom.config(dt), p, initial=True)
    o.step(1)
    a_scale, dr_scale = o.scales()
    ref = o.download()
    cfg = dom.config(dt)
    cfg.precision = precision
    gd = GpuDomain(cfg)
    gd.upload(p)
    gd.step(1)
    got = gd.download_fields(("a", "ddensity"))
    tol = 1e-5 if precision else 1e-12
    assert np.max(np.linalg.norm(got["a"] - ref["a"], axis=1)[free] / a_scale[free]) <= tol
    assert np.max(np.abs(got["ddensity"] - ref["ddensity"])[free] / (dr_scale[free] + 1e-300)) <= tol
    gd.close()
