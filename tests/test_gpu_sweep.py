"""The counted binning and the unit sweep of P2G and of its adjoint at the
layouts where they can go wrong: lanes without a particle, cells beyond the
ranking's 64 rows and across the 256-particle restarts, layers in rows and
cell after cell, units split in 4, 2 and 1 parts, cells at unit borders and
particles beside the grid's edge.

Bounds, with k the most particles of one cell and eps = 2^-24: a node's mass
and cubic sums add at most k float32 terms per cell, each with up to 8
roundings, on both sides (the cells' totals are exact here, float32 in the
oracle, whose running sum over 27 or more cells is of the same order): rel. L2
2 (k + 32) eps.  Momentum: 1e-5, the bound of one substep (its terms carry the
rounding of the eigensolve).  The adjoint: v' is affine in v and, with the damage
update at rest, lap' linear in d, so that the vector-Jacobian product has to
match the forward's own difference up to rounding: 2e-5 of the norms' product
(about 100 roundings on either side), for the Laplacian times the bound
12 / dx^2 of its weights.
"""
import numpy as np
import pytest
import torch

from helpers import make_gpu_sim, rel_l2
from test_gpu_parity import _rot, run_pieces, ws_views
import oracle as orc
from peel_mpm_b200 import scenes
import peel_mpm_b200.differentiable as dfx

pytestmark = pytest.mark.gpu


def _cell(rng, c, k, ng):
    return (np.asarray(c) + rng.uniform(0.55, 1.45, size=(k, 3))) / ng


def _layout(name, rng):
    """(n_grid, positions)"""
    if name == "one":
        return 16, _cell(rng, (7, 3, 8), 1, 16)
    if name == "cell of 64 and 65":                    # the ranking's last row and the first beyond
        ng = 24
        return ng, np.concatenate([_cell(rng, (8, 9, 7), 64, ng), _cell(rng, (8, 9, 8), 65, ng)])
    if name == "restarts":                             # 700 in a cell, 255, 1 and 2 around it: restarts at 256
        ng = 20
        return ng, np.concatenate([_cell(rng, (8, 8, 9), 700, ng), _cell(rng, (8, 8, 8), 255, ng),
                                   _cell(rng, (8, 9, 8), 1, ng), _cell(rng, (9, 8, 8), 2, ng)])
    if name == "rows":                                 # every cell of 3 x 2 x 2 units, 2 to 5 particles each
        ng = 33
        cells = np.stack(np.meshgrid(range(4, 16), range(8, 16), range(8, 24), indexing="ij"), -1).reshape(-1, 3)
        return ng, np.concatenate([_cell(rng, c, rng.integers(2, 6), ng) for c in cells])
    if name == "edge":                                 # base cells 0 .. n_grid - 2 along one axis, some outside
        ng = 19
        x = rng.uniform(0.0, 1.0, size=(1500, 3))
        x[:8] = [[-0.2, 0.5, 0.5], [1.3, 0.5, 0.5], [0.0, 0.0, 0.0], [1.0, 1.0, 1.0], [0.5, 0.5, 1.2],
                 [0.5, 1.01, 0.5], [0.02, 0.9, 0.3], [0.97, 0.02, 0.5]]
        return ng, x
    n = {"4 parts": 90, "2 parts": 200, "1 part": 2500}[name]   # units reached: <= 111, 112 .. 222, more
    ng = 64
    c = rng.permutation(14 * 14 * 7)[:min(n, 14 * 14 * 7)]
    c = np.stack([4 + 4 * (c // 98), 4 + 4 * (c // 7 % 14), 4 + 8 * (c % 7)], 1)   # one cell of each unit
    c = c + rng.integers(0, 3, size=c.shape)
    x = np.concatenate([_cell(rng, v, 1, ng) for v in c])
    return ng, np.concatenate([x, _cell(rng, (30, 30, 30), max(n - len(x), 7), ng)])


LAYOUTS = ["one", "cell of 64 and 65", "restarts", "rows", "edge", "4 parts", "2 parts", "1 part"]


def _scene(name):
    rng = np.random.default_rng(LAYOUTS.index(name) + 100)
    ng, x = _layout(name, rng)
    x = x[rng.permutation(len(x))].astype(np.float32).astype(np.float64)
    n = len(x)
    sc = scenes.Scene(name="sweep", n_grid=ng, grid_lim=1.0, dt=1e-4, n_steps=1, x=x, vol=rng.uniform(0.5e-6, 1e-6, n),
                      rho=800.0, E=np.full(n, 50.0), nu=0.3, fibers=None, alpha=0.0, sigma_c=np.full(n, 1e6),
                      d0=rng.uniform(0.0, 0.2, n), allow=np.ones(n, bool), gravity=(0.0, 0.0, 0.0))
    F = np.einsum("nij,nj,nkj->nik", _rot(rng, n), rng.uniform(0.9, 1.1, size=(n, 3)), _rot(rng, n))
    state = {"F": F, "v": rng.normal(size=(n, 3)), "C": rng.normal(size=(n, 3, 3))}
    # base cells as the solver computes them: most particles of one cell
    b = np.floor(x.astype(np.float32) * np.float32(ng) - np.float32(0.5)).astype(np.int64)
    k = int(np.unique(np.clip(b, 0, ng - 1), axis=0, return_counts=True)[1].max())
    return rng, sc, {f: a.astype(np.float32) for f, a in state.items()}, k


def _sim(sc, state):
    sim = make_gpu_sim(sc)
    for f, a in state.items():
        getattr(sim, f)[:] = torch.tensor(a, device="cuda:0")
    return sim


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
    tol = 2 * (k + 32) * 2.0 ** -24
    assert rel_l2(grids["grid_mv"], mom[:, :3]) < 1e-5
    assert rel_l2(grids["grid_m"], mom[:, 3]) < tol
    assert rel_l2(grids["grid_dc"], dmg[:, 0]) < tol
    assert rel_l2(grids["grid_dwc"], dmg[:, 1]) < tol
    # the same sums, bit for bit, once more from the state that the first substep left the workspace in
    raw = w["g_mom_raw"].clone(), w["g_dmg_raw"].clone()
    run_pieces(sim, 0.0, ("grid", "g2p"))
    again = _sim(sc, state)
    for _ in range(2):
        for f in ("x", "d", "lap", "D_hist"):
            getattr(again, f)[:] = getattr(_sim(sc, state), f)
        for f, a in state.items():
            getattr(again, f)[:] = torch.tensor(a, device="cuda:0")
        run_pieces(again, 0.0, ("bin", "p2g"))
        w = ws_views(again)
        assert torch.equal(w["g_mom_raw"], raw[0]) and torch.equal(w["g_dmg_raw"], raw[1])
        run_pieces(again, 0.0, ("grid", "g2p"))


@pytest.mark.parametrize("name", LAYOUTS)
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
