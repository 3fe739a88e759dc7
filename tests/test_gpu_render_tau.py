"""Depth weighting switched off: tau = infinity (and a float64 tau beyond float32, which becomes
infinite on the way) gives every splat the weight of its alpha alone, in the branch-free form (one
depth range per part of a tile) and in the general one."""
import numpy as np
import pytest
import torch

from peel_mpm_b200.render import Camera, render_gaussians
from test_gpu_render_parts import _image64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [float("inf"), 1e39, 3e38])
@pytest.mark.parametrize("odd", [False, True])            # a colour that is not finite: the general form
@pytest.mark.parametrize("n", [1, 33, 400])
def test_infinite_tau_matches_float64(n, odd, tau):
    """The renderer's image bound, 1e-4."""
    rng = np.random.default_rng(n)
    W, H, f, r_max = 50, 37, 40.0, 10
    z = rng.uniform(1.0, 9.0, n)
    xy = (rng.uniform(0.0, 1.0, (n, 2)) * [W, H] - [0.5 * W, 0.5 * H]) / f * z[:, None]
    R = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    size = (z / f)[:, None] * rng.uniform(0.4, 2.0, (n, 1)) * np.array([1.0, 0.7, 0.5])
    cov = (R * size[:, None, :] ** 2) @ R.transpose(0, 2, 1)
    xyz, cov, col = (a.astype(np.float32) for a in (np.c_[xy, z], cov, rng.uniform(0, 1, (n, 3))))
    if odd:                                               # on the image's last column, drawn by all parts' lists near it
        xyz[-1] = [(W - 0.5 - 0.5 * W) / f, 0.0, 1.0]
        cov[-1] = np.eye(3) * (0.1 / f) ** 2
        col[-1] = np.nan
    t = lambda a: torch.tensor(a, device="cuda:0")
    cam = Camera(R=np.eye(3), T=np.zeros(3), fx=f, fy=f, width=W, height=H, device="cuda:0")
    bg = (0.1, 0.2, 0.3)
    img = render_gaussians(cam, t(xyz), t(cov), t(col), t(np.ones(n, np.float32)), bg=bg, r_max=r_max, tau=tau)
    got = img.cpu().numpy()
    want = _image64(xyz, cov, col, f, W, H, tau, bg, r_max)
    left = slice(0, W - 4) if odd else slice(0, W)        # the odd splat's footprint: radius ceil(3 sqrt(0.31)) = 2
    assert np.abs(got[:, left] - want[:, left]).max() < 1e-4
    if n > 1:
        assert np.abs(got[:, left] - np.asarray(bg)).max() > 0.01
