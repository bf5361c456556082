"""FP32C, on a Shepard step: the filter's sums take a cell's particles slab by
slab and by original index inside a slab. With the particles uploaded by ascending
x that is the original order whatever the slabs, so the filtered sums and
densities have the same bits for every cell split, free particles and walls
together in a cell."""
import numpy as np
import pytest

from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain

pytestmark = pytest.mark.gpu


# (in 2D: ZWab of the 3D dam breaks, without the own term, stays below the filter's 0.6)
@pytest.mark.parametrize("kernel,hfac", [(0, 1.2), (2, 1.1)])
def test_split_independent(gpu, kernel, hfac):
    dx, dim = 0.031, 2
    dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.4, H=0.7, TL=1.1, TH=0.9, kernel=kernel, hfac=hfac)
    p = dom.particles
    p.set("shepard", 1)
    rng = np.random.default_rng(2)
    x = p.get("x")
    free = p.get("is_free") != 0
    x[free, :dim] += 0.2 * dx * (rng.random((int(free.sum()), dim)) - 0.5)
    p.set("x", x)
    order = np.argsort(x[:, 0], kind="stable")
    for f, a in p.arrays().items():
        p.arrays()[f] = np.ascontiguousarray(a[order])
    cfg = dom.config(dt)
    cfg.precision = 1
    ref = None
    for split in (1, 2, 4):
        it = GpuDomain(cfg).integrator()
        it.shepard_counter = cfg.shepard_step
        gd = GpuDomain(cfg, integ=it)
        gd.upload(p)
        gd.set_tuning(128, split)
        gd.step(1)
        got = gd.download_fields(("zwab", "sumden", "density"))
        gd.close()
        f = (p.get("is_free") != 0) & (got["zwab"] > 0.6)
        assert f.sum() > 100
        got = {k: a[f] for k, a in got.items()}
        if ref is None:
            ref = got
        for k in ref:
            np.testing.assert_array_equal(got[k], ref[k], err_msg=f"{k}, split {split}")
