"""Artificial viscosity changed for some particles only, by psph_patch between
two steps and by each host hook: every pair of the soil and solid kernels then
takes the mean of its two particles' coefficients. One step against the oracle
with the same particles, at the FP64 parity bound (1e-12 of each particle's sum
of term magnitudes)."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain
from tests.gpu_helpers import assert_step_parity

pytestmark = pytest.mark.gpu


def make(kind):
    if kind == "soil3d":
        dom, dt, _ = scenarios.granular_column_3d(dx=0.02, W=0.1, D=0.08, aspect=0.8, cohesion=1.0e3)
    else:
        dom, dt, _ = scenarios.granular_column(dx=0.02, aspect=0.8, cohesion=1.0e3)
    p = dom.particles
    if kind == "solid2d":
        p.set("material", 2)
        p.set("fail", 0)
        p.set("sigma", 0.0)
    rng = np.random.default_rng(3)
    free = p.get("is_free") != 0
    v = p.get("v")
    v[free, :dom.Dimension] += 0.5 * (rng.random((int(free.sum()), dom.Dimension)) - 0.5)  # approaching pairs
    p.set("v", v)
    return dom, dt


def unlike(p):
    """Another alpha for a third of the particles, another beta for a fifth."""
    i = np.arange(p.n)
    p.set("alpha", np.where(i % 3 == 0, 0.7, 0.1))
    p.set("beta", np.where(i % 5 == 0, 0.0, 0.1))


@pytest.mark.parametrize("how", ["patch", "before", "after"])
@pytest.mark.parametrize("kind", ["soil2d", "soil3d", "solid2d"])
def test_unlike_viscosity(gpu, kind, how):
    dom, dt = make(kind)
    cfg = dom.config(dt)
    gd = GpuDomain(cfg)
    if how == "after":
        gd.set_step_hooks(after=lambda t, p: unlike(p))
    gd.upload(dom.particles)
    gd.step(1)
    if how == "patch":
        p = gd.download()
        unlike(p)
        gd.patch(p)
    gd.set_step_hooks()
    state = gd.download()
    o = OracleDomain(cfg, state, initial=False, grid=gd.grid(), integ=gd.integrator())
    if how == "before":
        o.set_step_hooks(before=lambda t, p: unlike(p))
        gd.set_step_hooks(before=lambda t, p: unlike(p))
    assert how == "before" or len(np.unique(state.get("alpha"))) == 2
    o.step(1)
    gd.step(1)
    a_scale, dr_scale = o.scales()
    assert_step_parity(gd.download_fields(), o.download(), a_scale, dr_scale, dt, label=f"{kind} {how}")
    gd.close()
