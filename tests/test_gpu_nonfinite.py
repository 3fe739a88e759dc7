"""A particle whose momentum, or whose adjoint, is not a number or infinite: its cell's sums of that
quantity count for nothing in the fixed-point grid, as they always did, and nobody else is thrown
about.  (A conversion's result for such a sum is +-2^63 units, 2^17 times the largest contribution
there is: added to a node it would give every particle nearby a velocity of 1e5 and more.)

Bounds: the largest velocity after one substep without forces is at most the largest velocity of a
node, a mean of particle values v + C dpos, less what the dropped cell held: at most
(total / remaining mass) times, here below 8.  A factor of 20 is allowed for everything."""
import numpy as np
import pytest
import torch

from helpers import make_gpu_sim
from test_gpu_pieces import _scene
import peel_mpm_b200.differentiable as dfx

pytestmark = pytest.mark.gpu


def _sim(v):
    sc, _ = _scene()
    sc.E = np.full(sc.n, 1e-3)
    sc.gravity = (0.0, 0.0, 0.0)
    sim = make_gpu_sim(sc)
    sim.v[:] = v
    return sim


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("count", [1, 2, 5])
def test_momentum_that_is_not_finite_counts_for_nothing(bad, count):
    sc, v0 = _scene()
    v = torch.tensor(v0, device="cuda:0")
    who = torch.arange(count, device="cuda:0") * 801 + 77        # different cells
    v[who, 1] = bad
    sim = _sim(v)
    sim.substep(0.0)
    ok = torch.ones(sim.n, dtype=torch.bool, device="cuda:0")
    ok[who] = False
    got = sim.v[ok]
    assert torch.isfinite(got).all()
    assert float(got.abs().max()) < 20 * float(np.abs(v0).max())
    assert float((sim.x[ok] - torch.tensor(sc.x, device="cuda:0")[ok]).abs().max()) < 20 * sc.dt * float(np.abs(v0).max())


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_adjoint_that_is_not_finite_counts_for_nothing(bad):
    sc, v0 = _scene()
    v = torch.tensor(v0, device="cuda:0")
    w = torch.tensor(np.random.default_rng(2).normal(size=(sc.n, 3)).astype(np.float32), device="cuda:0")
    base = dfx.substep_vjp(_sim(v), 0.0, {"v": w})[0]["v"]
    w2 = w.clone()
    w2[777, 1] = bad
    got = dfx.substep_vjp(_sim(v), 0.0, {"v": w2})[0]["v"]
    ok = torch.ones(sc.n, dtype=torch.bool, device="cuda:0")
    ok[777] = False
    assert torch.isfinite(got[ok]).all()
    assert float(got[ok].abs().max()) < 20 * float(base.abs().max())
