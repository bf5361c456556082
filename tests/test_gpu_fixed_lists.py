"""Neighbour lists of fixed particles hold free particles only: a fixed particle
that a GeneralBefore hook frees (after the lists were made) still meets its
fixed neighbours in that step, as when it was freed before the step."""
import numpy as np
import pytest

from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuDomain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [1, 4])
@pytest.mark.parametrize("seed", [1, 2])
def test_freed_by_a_hook(gpu, seed, split):
    def make():
        dom, dt, _ = scenarios.dam_break_2d(dx=0.04, L=0.4, H=0.5, TL=0.9, TH=0.7)
        gd = GpuDomain(dom.config(dt))
        gd.upload(dom.particles)
        gd.set_tuning(128, split)
        return gd

    rng = np.random.default_rng(seed)
    a, b = make(), make()
    p = a.download()
    fixed = np.flatnonzero(p.get("is_free") == 0)
    pick = rng.choice(fixed, size=len(fixed) // 3, replace=False)

    def free(ps):
        f = ps.get("is_free").copy()
        f[pick] = 1
        ps.set("is_free", f)
        return ps

    a.patch(free(p))
    a.step(1)
    b.set_step_hooks(before=lambda t, ps: free(ps))
    b.step(1)
    fa, fb = a.download_fields(("a", "ddensity", "is_free")), b.download_fields(("a", "ddensity", "is_free"))
    assert fa["is_free"][pick].all() and fb["is_free"][pick].all()
    scale = np.abs(fa["a"]).max()
    assert np.abs(fa["a"] - fb["a"]).max() <= 1e-12 * scale
    assert np.abs(fa["ddensity"] - fb["ddensity"]).max() <= 1e-12 * np.abs(fa["ddensity"]).max() + 1e-300
    a.close()
    b.close()
