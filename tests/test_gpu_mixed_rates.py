"""Domains of two materials: downloaded rotation rates of fluid particles are zero,
and strain rates too unless the fluid sums them, also where a particle's sorted
place was a soil or solid particle's before; the others' are the oracle's."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,les", [("seepage", False), ("gate", False), ("gate", True)])
def test_rates_after_a_sort(gpu, kind, les):
    if kind == "seepage":
        dom, dt, _ = scenarios.seepage_bed_2d(dx=0.02, swi=0, cohesion=1.0e3)
    else:
        dom, dt, _ = scenarios.elastic_gate_2d(dx=0.01)
    dt *= 0.5
    p = dom.particles
    fluid = p.get("material") == 1
    if les:
        p.set("les", fluid.astype(np.int32))
        p.set("csmag", 0.17)
    free = p.get("is_free") != 0
    rng = np.random.default_rng(4)
    v = p.get("v")
    v[free, :2] += 0.5 * (rng.random((int(free.sum()), 2)) - 0.5)
    v[free, 0] += np.where(fluid[free], 1.5, -1.5)  # the materials drift past and into one another:
    v[free, 1] += np.where(fluid[free], -1.0, 1.0)  # places change hands
    p.set("v", v)
    cfg = dom.config(dt)
    gd = GpuDomain(cfg)
    gd.upload(p)
    gd.step(200)
    # (the last step alone: a yielding soil's trajectory takes rounding-level turns)
    o = OracleDomain(cfg, gd.download(), initial=False, grid=gd.grid(), integ=gd.integrator())
    o.step(1)
    gd.step(1)
    ref, got = o.download(), gd.download_fields(("strain_rate", "rotation_rate"))
    f = free & fluid
    assert not got["rotation_rate"][f].any()
    assert got["strain_rate"][f].any() == les
    for k in got:  # (the oracle keeps the rates it was given where it sums none)
        sel = free if k == "strain_rate" and les else free & ~fluid
        assert np.abs(got[k] - ref[k])[sel].max() <= 1e-9 * np.abs(ref[k][sel]).max(), k
    gd.close()
