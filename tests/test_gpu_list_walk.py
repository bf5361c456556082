"""The two-particle list scan walks a row's three cells in groups of four
candidates, the last group of a cell partly masked: cells of every fill from
empty upwards (a shaken lattice), cell splits, the staged copy, and a tall
support, one step against the oracle at the FP64 form's parity bound."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain
from tests.gpu_helpers import assert_step_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split,stage", [(1, 0), (2, 0), (4, 0), (1, 3072), (4, 4096)])
@pytest.mark.parametrize("dim,hfac", [(2, 1.2), (2, 2.2), (3, 1.3)])
def test_shaken_lattice(gpu, dim, hfac, split, stage):
    dx = 0.05
    if dim == 2:
        dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.5, H=0.65, TL=1.0, TH=0.8, hfac=hfac)
    else:
        dom, dt, _ = scenarios.dam_break_3d(dx=dx, L=0.3, H=0.35, W=0.25, TL=0.5, TH=0.4, TW=0.25, hfac=hfac)
    p = dom.particles
    rng = np.random.default_rng(7)
    free = p.get("is_free") != 0
    x = p.get("x")
    x[free, :dim] += 0.6 * dx * (rng.random((int(free.sum()), dim)) - 0.5)
    p.set("x", x)
    cfg = dom.config(dt)
    o = OracleDomain(cfg, p, initial=True)
    gd = GpuDomain(cfg)
    gd.upload(p)
    gd.set_tuning(128, split, stage)
    assert set(map(tuple, gd.pairs(1).tolist())) == set(map(tuple, o.pairs(3).tolist()))
    o.step(1)
    gd.step(1)
    a_scale, dr_scale = o.scales()
    assert_step_parity(gd.download_fields(), o.download(), a_scale, dr_scale, dt, label=f"{dim}D {hfac} {split} {stage}")
    gd.close()
