"""The pieces of a substep through the C ABI out of step: a P2G whose grid update never runs, as a
caller makes it to look at the grid sums, and two P2Gs under one clock.  Later substeps must update
every block they touch.

What such a P2G leaves behind is the node sums, which the next one adds to: momentum, mass and
damage sums double, exactly, and the velocities and damage that the grid update divides out of them
stay the same up to rounding: 1e-6, a few eps."""
import numpy as np
import pytest
import torch

from helpers import FIELDS, make_gpu_sim, rel_l2
from test_gpu_parity import run_pieces
from peel_mpm_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(ng=24):
    rng = np.random.default_rng(5)
    ax = np.arange(8, 16)
    c = np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 1, 3)
    s = (np.stack(np.meshgrid(*[range(2)] * 3, indexing="ij"), -1).reshape(1, 8, 3) + 0.5) / 2
    x = ((c + s).reshape(-1, 3) / ng).astype(np.float32).astype(np.float64)
    n = len(x)
    sc = scenes.Scene(name="pieces", n_grid=ng, grid_lim=1.0, dt=1e-4, n_steps=1, x=x, vol=np.full(n, 1e-5),
                      rho=800.0, E=np.full(n, 1e3), nu=0.3, fibers=None, alpha=0.0, sigma_c=np.full(n, 1e2),
                      d0=rng.uniform(0.0, 0.2, n), allow=np.ones(n, bool), gravity=(0.0, -9.8, 0.0))
    return sc, rng.normal(size=(n, 3)).astype(np.float32)


@pytest.mark.parametrize("before", [("bin", "p2g"), ("bin", "p2g", "p2g"), ("bin", "p2g", "bin", "p2g")])
@pytest.mark.parametrize("then", ["substeps", "frame", "pieces"])
def test_unfinished_substep_does_not_spoil_the_next(before, then):
    sc, v = _scene()
    sims = []
    for k in range(2):
        sim = make_gpu_sim(sc)
        sim.v[:] = torch.tensor(v, device="cuda:0")
        if k:
            d, D = sim.d.clone(), sim.D_hist.clone()
            for stage in before:
                run_pieces(sim, 0.0, (stage,))
                sim.d[:], sim.D_hist[:] = d, D            # P2G's own state update is not part of the question
        if then == "substeps":
            for i in range(3):
                sim.substep(i * sc.dt)
        elif then == "frame":
            sim.run_frame(3, 0.0)
        else:
            for i in range(3):
                run_pieces(sim, i * sc.dt, ("bin", "p2g", "grid", "g2p"))
        sims.append(sim)
    for f in FIELDS:
        assert rel_l2(getattr(sims[0], f).cpu().numpy(), getattr(sims[1], f).cpu().numpy()) < 1e-6, f


def test_two_p2gs_under_one_clock_list_every_block_once():
    sc, v = _scene()
    sims = []
    for stages in (("bin", "p2g", "grid", "g2p"), ("bin", "p2g", "p2g", "grid", "g2p")):
        sim = make_gpu_sim(sc)
        sim.v[:] = torch.tensor(v, device="cuda:0")
        sim.allow[:] = False                              # damage at rest: the second P2G repeats the first
        for s in stages:
            run_pieces(sim, 0.0, (s,))
        sims.append(sim)
    for f in FIELDS:
        assert rel_l2(getattr(sims[0], f).cpu().numpy(), getattr(sims[1], f).cpu().numpy()) < 1e-6, f
