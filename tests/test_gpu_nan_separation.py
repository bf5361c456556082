"""A position that is not a number, written by a GeneralBefore hook after the
neighbour lists are made, ends the step as non-finite, whatever the NaN's sign:
FP64 and FP32C, fluid and soil, every kernel."""
import numpy as np
import pytest

from persiansph_gb300 import scenarios
from persiansph_gb300.abi import PsphError
from persiansph_gb300.solver import GpuDomain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind,kernel", [("fluid", 0), ("fluid", 1), ("fluid", 2), ("les", 0), ("soil", 0)])
def test_nan_position(gpu, kind, kernel, precision, sign):
    if kind == "soil":
        dom, dt, _ = scenarios.granular_column(dx=0.02, aspect=0.8, cohesion=1.0e3)
    else:
        dom, dt, _ = scenarios.dam_break_2d(dx=0.04, L=0.4, H=0.5, TL=0.9, TH=0.7, kernel=kernel)
    p = dom.particles
    if kind == "les":
        p.set("les", 1)
        p.set("csmag", 0.17)
    free = np.flatnonzero(p.get("is_free") != 0)
    cfg = dom.config(dt)
    cfg.precision = precision
    gd = GpuDomain(cfg)

    def hook(t, s):
        x = s.get("x")
        x[free[len(free) // 2], 0] = np.copysign(np.nan, sign)
        s.set("x", x)

    gd.set_step_hooks(before=hook)
    gd.upload(p)
    with pytest.raises(PsphError) as e:
        gd.step(1)
    assert "non-finite" in str(e.value)
    gd.close()
