"""The counted binning: every particle's payload place, read back, runs in id order within its cell
whatever the cell holds (columns of 64, sorted runs of 512, several runs, and the start's headroom
and beyond), and the unit sweep's list at the length where it changes from single layers to whole
units, one item more and one less.

Bounds of the sums as in test_gpu_sweep; places are whole numbers."""
import numpy as np
import pytest
import torch

from helpers import rel_l2
from test_gpu_parity import _rot, run_pieces, ws_views
from test_gpu_sweep import _cell, _sim
import oracle as orc
from peel_mpm_b200 import _lib, scenes
import peel_mpm_b200.differentiable as dfx

pytestmark = pytest.mark.gpu


def _scene(ng, x, seed):
    rng = np.random.default_rng(seed)
    x = x[rng.permutation(len(x))].astype(np.float32).astype(np.float64)
    n = len(x)
    sc = scenes.Scene(name="binning", n_grid=ng, grid_lim=1.0, dt=1e-4, n_steps=1, x=x,
                      vol=rng.uniform(0.5e-6, 1e-6, n), rho=800.0, E=np.full(n, 50.0), nu=0.3, fibers=None, alpha=0.0,
                      sigma_c=np.full(n, 1e6), d0=rng.uniform(0.0, 0.2, n), allow=np.ones(n, bool))
    return sc, {"v": rng.normal(size=(n, 3)).astype(np.float32)}


def _places(sim):
    """w.slot: after the work list of n ints in the workspace."""
    L = _lib.workspace_layout(sim.n, sim.n_grid)
    off = L.work + (4 * sim.n + 255) // 256 * 256
    return sim._ws[off:off + 4 * sim.n].view(torch.int32).cpu().numpy().astype(np.int64)


@pytest.mark.parametrize("counts", [(1, 2, 31), (63, 64, 65), (511, 512, 513), (1023, 1024, 1025), (3000, 700, 64),
                                    (65532, 65533, 5), (150001, 1, 0)])
@pytest.mark.parametrize("edge", [False, True])
def test_places_run_in_id_order(counts, edge):
    rng = np.random.default_rng(sum(counts))
    ng = 20
    cells = [(0, 8, 9), (0, 8, 10), (0, 9, 9)] if edge else [(8, 8, 9), (8, 8, 10), (8, 9, 9)]
    x = np.concatenate([_cell(rng, c, k, ng) for c, k in zip(cells, counts)] +
                       [_cell(rng, (8 + i % 3, 12 + i // 9 % 3, 4 + i // 3 % 3), 3, ng) for i in range(27)])
    sc, state = _scene(ng, x, 7)
    sim = _sim(sc, state)
    run_pieces(sim, 0.0, ("bin", "p2g"))
    at = _places(sim)
    assert len(np.unique(at)) == sc.n and at.min() >= 0 and at.max() < (2 * sc.n + 31) // 32 * 32
    b = np.clip(np.floor(sc.x.astype(np.float32) * np.float32(ng) - np.float32(0.5)), 0, ng - 1).astype(np.int64)
    key = (b[:, 0] * ng + b[:, 1]) * ng + b[:, 2]
    order = np.lexsort((np.arange(sc.n), key))
    same = key[order][1:] == key[order][:-1]
    assert (np.diff(at[order])[same] > 0).all()


@pytest.mark.parametrize("more", [-1, 0, 1, 40])
def test_sums_at_the_border_of_single_layers(more):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ng, units = 64, sms + more                          # one CTA per SM below: units == CTAs is the border
    rng = np.random.default_rng(units)
    c = rng.permutation(14 * 14 * 7)[:units]
    c = np.stack([4 + 4 * (c // 98), 4 + 4 * (c // 7 % 14), 4 + 8 * (c % 7)], 1)
    x = np.concatenate([_cell(rng, v + rng.integers(0, 3, 3), 1 + i % 5, ng) for i, v in enumerate(np.repeat(c, 3, 0))])
    sc, state = _scene(ng, x, 3)
    F = np.einsum("nij,nj,nkj->nik", _rot(rng, sc.n), rng.uniform(0.9, 1.1, size=(sc.n, 3)), _rot(rng, sc.n))
    state.update(F=F.astype(np.float32), C=rng.normal(size=(sc.n, 3, 3)).astype(np.float32))
    ora = orc.OracleSim(sc, np.float32)
    for f, a in state.items():
        getattr(ora, f)[:] = a
    grids = ora.alloc_grids()
    ora.substep(0.0, grids=grids)
    sim = _sim(sc, state)
    sim.p2g_ctas_per_sm = 1
    run_pieces(sim, 0.0, ("bin", "p2g"))
    w = ws_views(sim)
    mom, dmg = w["g_mom"].cpu().numpy().astype(np.float64), w["g_dmg"].cpu().numpy().astype(np.float64)
    tol = 2 * (16 + 32) * 2.0 ** -24
    assert rel_l2(grids["grid_mv"], mom[:, :3]) < 1e-5
    for got, name in ((mom[:, 3], "grid_m"), (dmg[:, 0], "grid_dc"), (dmg[:, 1], "grid_dwc")):
        assert rel_l2(grids[name], got) < tol


def _cloud():
    """Fewer than 24 particles to a unit: layers of one and two cells add cell by cell, three go the general way; among
    them cells of 256 and 300, which restart at 256."""
    ng = 64
    rng = np.random.default_rng(11)
    c = rng.permutation(14 * 14 * 7)[:80]
    c = np.stack([4 + 4 * (c // 98), 4 + 4 * (c // 7 % 14), 4 + 8 * (c % 7)], 1)
    x = [_cell(rng, v, 256 if i == 0 else 300, ng) for i, v in enumerate(c[:2])]
    for i, v in enumerate(c[2:]):
        for k in range(1 + i % 3):                      # cells of one layer
            x.append(_cell(rng, v + [0, k, 2 * k], 1 + i % 4, ng))
    sc, state = _scene(ng, np.concatenate(x), 5)
    assert sc.n < 24 * 80
    F = np.einsum("nij,nj,nkj->nik", _rot(rng, sc.n), rng.uniform(0.9, 1.1, size=(sc.n, 3)), _rot(rng, sc.n))
    state.update(F=F.astype(np.float32), C=rng.normal(size=(sc.n, 3, 3)).astype(np.float32))
    return rng, sc, state


def test_sums_of_a_cloud_match_the_oracle():
    rng, sc, state = _cloud()
    ora = orc.OracleSim(sc, np.float32)
    for f, a in state.items():
        getattr(ora, f)[:] = a
    grids = ora.alloc_grids()
    ora.substep(0.0, grids=grids)
    sim = _sim(sc, state)
    run_pieces(sim, 0.0, ("bin", "p2g"))
    w = ws_views(sim)
    mom, dmg = w["g_mom"].cpu().numpy().astype(np.float64), w["g_dmg"].cpu().numpy().astype(np.float64)
    tol = 2 * (300 + 32) * 2.0 ** -24
    assert rel_l2(grids["grid_mv"], mom[:, :3]) < max(1e-5, tol)
    for got, name in ((mom[:, 3], "grid_m"), (dmg[:, 0], "grid_dc"), (dmg[:, 1], "grid_dwc")):
        assert rel_l2(grids[name], got) < tol


def test_vjp_of_a_cloud_matches_the_forward_differences():
    rng, sc, state = _cloud()
    w = torch.tensor(rng.normal(size=(sc.n, 3)), dtype=torch.float32, device="cuda:0")
    wl = torch.tensor(rng.normal(size=sc.n), dtype=torch.float32, device="cuda:0")

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
