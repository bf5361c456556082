"""The neighbour-list scans on cells of every fill from empty upwards (a shaken
lattice), one step against the oracle at the FP64 form's parity bound: a lane to
a cell (few particles), the walk of a row's three cells in groups of four with
the last of a cell partly masked (many, or the staged copy), cell splits, a tall
support, cells fuller than a lane's bits, and a grid whose bins take more than
one launch to scan."""
import numpy as np
import pytest

from oracle.oracle import OracleDomain
from persiansph_gb300 import scenarios
from persiansph_gb300.solver import GpuEnsemble, GpuDomain
from tests.gpu_helpers import assert_step_parity

pytestmark = pytest.mark.gpu


def shaken(p, dx, dim, by=0.6, seed=7):
    rng = np.random.default_rng(seed)
    free = p.get("is_free") != 0
    x = p.get("x")
    x[free, :dim] += by * dx * (rng.random((int(free.sum()), dim)) - 0.5)
    p.set("x", x)


def one_step(dom, dt, label, tuning=None):
    cfg = dom.config(dt)
    o = OracleDomain(cfg, dom.particles, initial=True)
    gd = GpuDomain(cfg)
    gd.upload(dom.particles)
    if tuning:
        gd.set_tuning(128, *tuning)
    assert set(map(tuple, gd.pairs(1).tolist())) == set(map(tuple, o.pairs(3).tolist()))
    o.step(1)
    gd.step(1)
    a_scale, dr_scale = o.scales()
    assert_step_parity(gd.download_fields(), o.download(), a_scale, dr_scale, dt, label=label)
    gd.close()


@pytest.mark.parametrize("split,stage", [(1, 0), (2, 0), (4, 0), (1, 3072), (4, 4096)])
@pytest.mark.parametrize("dim,hfac", [(2, 1.2), (2, 2.2), (3, 1.3)])
def test_shaken_lattice(gpu, dim, hfac, split, stage):
    dx = 0.05
    if dim == 2:
        dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.5, H=0.65, TL=1.0, TH=0.8, hfac=hfac)
    else:
        dom, dt, _ = scenarios.dam_break_3d(dx=dx, L=0.3, H=0.35, W=0.25, TL=0.5, TH=0.4, TW=0.25, hfac=hfac)
    shaken(dom.particles, dx, dim)
    one_step(dom, dt, f"{dim}D {hfac} {split} {stage}", (split, stage))


@pytest.mark.parametrize("dim,split", [(2, 1), (2, 4), (3, 1), (3, 4)])
def test_more_than_the_lanes_to_a_cell(gpu, dim, split):  # a lane to a particle
    if dim == 2:
        dx = 0.01
        dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=1.2, H=1.6, TL=2.0, TH=2.0)
    else:
        dx = 0.03
        dom, dt, _ = scenarios.dam_break_3d(dx=dx, L=0.7, H=0.5, W=0.6, TL=1.0, TH=0.6, TW=0.6)
    assert dom.particles.n > 152 * 2048 >> (4 if dim == 2 else 5)
    shaken(dom.particles, dx, dim)
    one_step(dom, dt, f"{dim}D split {split}", (split, 0))


def test_cells_fuller_than_a_lanes_bits(gpu):
    dx = 0.05
    dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=1.0, H=1.0, TL=1.4, TH=1.2, hfac=4.5)  # 9 x 9 particles to a cell
    shaken(dom.particles, dx, 2, 0.2)
    one_step(dom, dt, "full cells")


@pytest.mark.parametrize("split", [1, 4])
def test_sparse_grid(gpu, split):
    dx = 0.05
    dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.5, H=0.65, TL=16.5, TH=16.5)
    shaken(dom.particles, dx, 2)
    one_step(dom, dt, f"sparse {split}", (split, 0))


@pytest.mark.parametrize("dim,split", [(2, 1), (2, 4), (3, 1)])
def test_two_particles_to_a_lane(gpu, dim, split):
    """Many instances (two particles to a lane) give each the bits it has alone
    (a lane to a cell, or to a particle): the same lists in the same order."""
    dx = 0.02 if dim == 2 else 0.04
    doms = []
    for seed in range(3):
        if dim == 2:
            dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=1.2, H=1.6, TL=2.0, TH=2.0)
        else:
            dom, dt, _ = scenarios.dam_break_3d(dx=dx, L=0.7, H=0.5, W=0.6, TL=1.0, TH=0.6, TW=0.6)
        shaken(dom.particles, dx, dim, seed=seed)
        doms.append(dom)
    copies = 152 * 2048 // (3 * doms[0].particles.n) + 2
    assert 3 * copies * doms[0].particles.n > 152 * 2048
    b = GpuEnsemble([doms[q % 3].config(dt) for q in range(3 * copies)])
    b.upload([doms[q % 3].particles for q in range(3 * copies)])
    b.set_tuning(128, split)
    b.step(2)
    for seed, q in ((0, 0), (1, 3 * copies - 2), (2, 3 * copies // 2 // 3 * 3 + 2)):
        g = GpuDomain(doms[seed].config(dt))
        g.upload(doms[seed].particles)
        g.set_tuning(128, split)
        g.step(2)
        one, many = g.download_fields(("x", "v", "density", "a")), b.download_fields(q, ("x", "v", "density", "a"))
        for f in one:
            assert np.array_equal(one[f], many[f]), f
        g.close()
    b.close()


@pytest.mark.parametrize("dx,split", [(0.05, 1), (0.05, 4), (0.01, 2)])
def test_unlike_smoothing_lengths(gpu, dx, split):  # a lane to a cell, and to a particle
    dom, dt, _ = scenarios.dam_break_2d(dx=dx, L=0.5 if dx > 0.02 else 1.2, H=0.65 if dx > 0.02 else 1.6, TL=2.0, TH=2.0)
    p = dom.particles
    shaken(p, dx, 2)
    h = p.get("h")
    h *= 1.0 + 0.15 * np.random.default_rng(9).random(len(h))
    p.set("h", h)
    one_step(dom, dt, f"h, dx {dx}", (split, 0))
