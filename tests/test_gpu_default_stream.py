"""A context's work does not depend on the default stream: with that stream busy
(a bounded spin of a tenth of a second from another library), upload, steps, row
counts, downloads, closure attachment and snapshots give the bits they give
alone. (A context's stream does not wait for the default one, so memory zeroed
there could lose what the context had written.)"""
import numpy as np
import pytest

from persiansph_gb300 import scenarios
from persiansph_gb300.closure import ClosureNet, default_network_path, les_case
from persiansph_gb300.solver import GpuDomain, GpuEnsemble

pytestmark = pytest.mark.gpu

FIELDS = ("x", "v", "density", "a", "ddensity", "sigma", "strain_rate")


def case(kind):
    if kind == "soil":
        return scenarios.granular_column(dx=0.02, aspect=0.8, cohesion=1.0e3)[:2]
    if kind == "les":
        return les_case(0.05, L=0.3, H=0.35, W=0.25, TL=0.6, TH=0.4, TW=0.25)[:2]
    return scenarios.dam_break_2d(dx=0.04, L=0.4, H=0.6, TL=1.0, TH=0.8)[:2]


def run(kind, precision, busy):
    dom, dt = case(kind)
    cfg = dom.config(dt)
    cfg.precision = precision
    busy()
    gd = GpuDomain(cfg)
    gd.upload(dom.particles)
    if kind == "les":
        net = ClosureNet.load(default_network_path())
        busy()
        gd.attach_closure(net, 0.05)
    gd.step(3)
    busy()
    n = gd.n
    busy()
    out = gd.download_fields(FIELDS)
    out["index"] = gd.original_index()
    out["pairs"] = np.sort(gd.pairs(1), axis=0)
    gd.close()
    assert n == dom.particles.n
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["fluid", "soil", "les"])
def test_busy_default_stream(gpu, kind, precision):
    torch = pytest.importorskip("torch")
    alone = run(kind, precision, lambda: None)
    torch.cuda.synchronize()
    got = run(kind, precision, lambda: torch.cuda._sleep(200_000_000))
    torch.cuda.synchronize()
    for k in alone:
        np.testing.assert_array_equal(got[k], alone[k], err_msg=k)


def test_busy_default_stream_ensemble(gpu):
    torch = pytest.importorskip("torch")
    doms = [scenarios.dam_break_2d(dx=0.04, L=0.4, H=0.6, TL=1.0, TH=0.8, alpha=a)[:2] for a in (0.1, 0.3)]

    def run_all(busy):
        busy()
        ens = GpuEnsemble([d.config(0.2 * dt) for d, dt in doms])
        ens.upload([d.particles for d, _ in doms])
        ens.step(3)
        busy()
        out = [ens.download_fields(q, FIELDS) for q in range(2)]
        ens.close()
        return out

    alone = run_all(lambda: None)
    torch.cuda.synchronize()
    got = run_all(lambda: torch.cuda._sleep(200_000_000))
    torch.cuda.synchronize()
    for a, g in zip(alone, got):
        for k in a:
            np.testing.assert_array_equal(g[k], a[k], err_msg=k)
