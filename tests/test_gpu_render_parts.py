"""The renderer's median by selection and its tile lists, at the
sizes where they can go wrong: one key, ties, a key set that shares its leading
digits, a rank on a digit's border, undrawn splats, and images of one tile up
to many CTAs of them."""
import numpy as np
import pytest
import torch

from peel_mpm_b200.render import Camera, render_gaussians

pytestmark = pytest.mark.gpu


def _cloud(z, W, H, f, seed):
    """Splats of depth z (behind the camera where negative), about 1 pixel wide, on the image."""
    rng = np.random.default_rng(seed)
    n = len(z)
    x = (rng.uniform(0, W, n) - 0.5 * W) / f * z
    y = (rng.uniform(0, H, n) - 0.5 * H) / f * z
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda:0")
    cov = np.eye(3)[None] * (np.abs(z) / f)[:, None, None] ** 2
    cam = Camera(R=np.eye(3), T=np.zeros(3), fx=float(f), fy=float(f), width=W, height=H, device="cuda:0")
    return cam, t(np.stack([x, y, z], 1)), t(cov), t(rng.uniform(0, 1, (n, 3))), t(np.ones(n))


@pytest.mark.parametrize("n,kind,W,H", [(1, "spread", 8, 8), (2, "spread", 8, 8), (33, "ties", 17, 9),
                                        (256, "close", 64, 40), (1025, "spread", 320, 200), (4099, "behind", 333, 77),
                                        (150_001, "close", 640, 480), (3000, "border", 1400, 1000)])
def test_median_tau_equals_the_given_one(n, kind, W, H):
    """tau from the depths gives the image of tau = 0.02 x the sorted depths' lower
    middle.  Only the order of the tile lists differs between the two calls: every
    pixel's sums have at most a few thousand float32 terms of one sign, 1e-4 is
    the renderer's image bound."""
    rng = np.random.default_rng(n)
    z = rng.uniform(0.5, 8.0, n)
    if kind == "ties":
        z = rng.choice([1.0, 1.5, 2.0], n)
    if kind == "close":                                   # the same exponent and leading mantissa bits
        z = 1.0 + 1e-4 * rng.random(n)
    if kind == "behind":
        z[::3] *= -1.0
    if kind == "border":                                  # the rank lands on the first key of a new digit
        z = np.where(np.arange(n) < (n - 1) // 2, 0.9999, 2.0)
    z = z.astype(np.float32).astype(np.float64)
    cam, xyz, cov, col, op = _cloud(z, W, H, 0.8 * W, n)
    drawn = np.sort(z[z > 0].astype(np.float32))
    tau = float(np.float32(0.02) * drawn[(len(drawn) - 1) // 2])
    a = render_gaussians(cam, xyz, cov, col, op, bg=(0.1, 0.2, 0.3))
    b = render_gaussians(cam, xyz, cov, col, op, bg=(0.1, 0.2, 0.3), tau=tau)
    assert float((a - b).abs().max()) < 1e-4
    assert float((a - torch.tensor([0.1, 0.2, 0.3], device="cuda:0")).abs().max()) > 0.01
