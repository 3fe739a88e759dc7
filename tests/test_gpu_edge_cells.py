"""Cells whose stencils need the reference's clamped nodes (base cell outside [1, n_grid - 4]), in P2G
and in its adjoint: a body resting on the upper end of the domain, crowded cells on faces, edges and
corners, runs of 32 particles and one more, and positions outside the domain, whose base cells
differ though they share a cell of the table.

Bounds as for the sweep (test_gpu_sweep): sums of up to k float32 terms of a cell, each with up to 8
roundings, against float32 sums in the oracle: rel. L2 2 (k + 32) 2^-24, momentum 1e-5; the adjoint
against the forward's own difference, 2e-5 of the norms' product."""
import numpy as np
import pytest
import torch

from helpers import rel_l2
from test_gpu_parity import _rot, run_pieces, ws_views
from test_gpu_sweep import _cell, _sim
import oracle as orc
from peel_mpm_b200 import scenes
import peel_mpm_b200.differentiable as dfx

pytestmark = pytest.mark.gpu


def _layout(name, rng):
    if name == "resting":                              # lattice cells up to base n_grid - 3, the last half filled
        ng = 21
        c = np.stack(np.meshgrid(range(6, 14), range(ng - 8, ng - 2), range(5, 16), indexing="ij"), -1).reshape(-1, 3)
        x = np.concatenate([_cell(rng, v, 8, ng) for v in c])
        x[:, 1] = np.minimum(x[:, 1], (ng - 2) / ng)
        return ng, x
    if name == "runs":                                 # 31, 32, 33 and 65 particles in cells of one layer and beside it
        ng = 16
        return ng, np.concatenate([_cell(rng, (0, 5, 5), 31, ng), _cell(rng, (0, 5, 6), 32, ng),
                                   _cell(rng, (0, 6, 5), 33, ng), _cell(rng, (0, 6, 6), 65, ng),
                                   _cell(rng, (ng - 3, 6, 6), 1, ng), _cell(rng, (1, 6, 6), 9, ng)])
    if name == "corners":
        ng = 12
        c = [(a, b, d) for a in (0, ng - 3) for b in (0, 5, ng - 3) for d in (0, ng - 2)]
        return ng, np.concatenate([_cell(rng, v, 40, ng) for v in c])
    if name == "outside":                              # far and near outside, every axis; some inside
        ng = 14
        x = rng.uniform(-0.6, 1.6, size=(700, 3))
        x[:4] = [[-50.0, 0.5, 0.5], [0.5, 1e4, 0.5], [-1e6, 1e6, 0.5], [0.5, 0.5, -3.0]]
        return ng, x
    if name == "small grid":                           # no regular cell but one
        return 5, rng.uniform(0.0, 1.0, size=(300, 3))
    return 4, rng.uniform(0.0, 1.0, size=(100, 3))     # none at all


LAYOUTS = ["resting", "runs", "corners", "outside", "small grid", "smallest grid"]


def _scene(name):
    rng = np.random.default_rng(LAYOUTS.index(name) + 500)
    ng, x = _layout(name, rng)
    x = x[rng.permutation(len(x))].astype(np.float32).astype(np.float64)
    n = len(x)
    sc = scenes.Scene(name="edge", n_grid=ng, grid_lim=1.0, dt=1e-4, n_steps=1, x=x, vol=rng.uniform(0.5e-6, 1e-6, n),
                      rho=800.0, E=np.full(n, 50.0), nu=0.3, fibers=None, alpha=0.0, sigma_c=np.full(n, 1e6),
                      d0=rng.uniform(0.0, 0.2, n), allow=np.ones(n, bool), gravity=(0.0, 0.0, 0.0))
    F = np.einsum("nij,nj,nkj->nik", _rot(rng, n), rng.uniform(0.9, 1.1, size=(n, 3)), _rot(rng, n))
    state = {"F": F, "v": rng.normal(size=(n, 3)), "C": rng.normal(size=(n, 3, 3))}
    b = np.clip(np.floor(x * ng - 0.5), 0, ng - 1).astype(np.int64)
    k = int(np.unique(b, axis=0, return_counts=True)[1].max())
    return rng, sc, {f: a.astype(np.float32) for f, a in state.items()}, k


@pytest.mark.parametrize("name", LAYOUTS)
def test_grid_sums_match_the_oracle(name):
    rng, sc, state, k = _scene(name)
    ora = orc.OracleSim(sc, np.float32)
    for f, a in state.items():
        getattr(ora, f)[:] = a
    sim = _sim(sc, state)
    grids = ora.alloc_grids()
    ora.substep(0.0, grids=grids)
    run_pieces(sim, 0.0, ("bin", "p2g"))
    w = ws_views(sim)
    mom, dmg = w["g_mom"].cpu().numpy().astype(np.float64), w["g_dmg"].cpu().numpy().astype(np.float64)
    if name == "outside":
        k = sc.n                                       # all that lies outside on one side meets in a few nodes
    tol = 2 * (k + 32) * 2.0 ** -24
    assert rel_l2(grids["grid_mv"], mom[:, :3]) < max(1e-5, tol)
    assert rel_l2(grids["grid_m"], mom[:, 3]) < tol
    assert rel_l2(grids["grid_dc"], dmg[:, 0]) < tol
    assert rel_l2(grids["grid_dwc"], dmg[:, 1]) < tol


@pytest.mark.parametrize("name", ["resting", "runs", "corners", "small grid", "smallest grid"])
def test_vjp_matches_the_forward_differences(name):
    rng, sc, state, _ = _scene(name)
    n = sc.n
    w = torch.tensor(rng.normal(size=(n, 3)), dtype=torch.float32, device="cuda:0")
    wl = torch.tensor(rng.normal(size=n), dtype=torch.float32, device="cuda:0")

    def forward(v, d):
        sim = _sim(sc, state)
        sim.v[:], sim.d[:] = v, d
        sim.substep(0.0)
        return sim.v.double(), sim.lap.double()

    u, d = torch.tensor(state["v"], device="cuda:0"), _sim(sc, state).d.clone()
    got = dfx.substep_vjp(_sim(sc, state), 0.0, {"v": w})[0]["v"].double()
    want = (w.double() * (forward(u, d)[0] - forward(0 * u, d)[0])).sum()
    assert abs(float((got * u).sum() - want)) < 2e-5 * float(w.norm() * u.norm())
    got = dfx.substep_vjp(_sim(sc, state), 0.0, {"lap": wl})[0]["d"].double()
    want = (wl.double() * (forward(u, d)[1] - forward(u, 0 * d)[1])).sum()
    assert abs(float((got * d).sum() - want)) < 2e-5 * float(wl.norm() * d.norm()) * 12 * sc.n_grid ** 2
