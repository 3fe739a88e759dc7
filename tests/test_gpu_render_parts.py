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


def _image64(xyz, cov, col, f, W, H, tau, bg, r_max, near=0.05):
    """render.py's image of a camera at the origin, in float64."""
    X, z = xyz.astype(np.float64), xyz[:, 2].astype(np.float64)
    ok = z > near
    zs = np.where(ok, z, 1.0)
    u, v = f * X[:, 0] / zs + 0.5 * W, f * X[:, 1] / zs + 0.5 * H
    J = np.zeros((len(z), 2, 3))
    J[:, 0, 0] = J[:, 1, 1] = f / zs
    J[:, 0, 2], J[:, 1, 2] = -f * X[:, 0] / zs ** 2, -f * X[:, 1] / zs ** 2
    S = J @ cov.astype(np.float64) @ J.transpose(0, 2, 1) + 0.3 * np.eye(2)
    lam = np.linalg.eigvalsh(S)[:, 1]
    rad = np.clip(np.ceil(3 * np.sqrt(lam)), 1, r_max)
    Q = np.linalg.inv(S)
    py, px = np.mgrid[0:H, 0:W]
    csum, wsum, zmin = np.zeros((H, W, 3)), np.zeros((H, W)), np.full((H, W), np.inf)
    rest, shown = np.ones((H, W)), []
    for i in np.flatnonzero(ok):
        dx, dy = px + 0.5 - u[i], py + 0.5 - v[i]
        p = -0.5 * (Q[i, 0, 0] * dx * dx + Q[i, 1, 1] * dy * dy) - Q[i, 0, 1] * dx * dy
        a = np.exp(np.minimum(p, 0.0))
        a[(np.abs(px - np.floor(u[i])) > rad[i]) | (np.abs(py - np.floor(v[i])) > rad[i]) | (a <= 1 / 255)] = 0.0
        shown.append((i, a))
        zmin = np.where(a > 0, np.minimum(zmin, z[i]), zmin)
        rest *= np.maximum(1.0 - a, 1e-6)
    for i, a in shown:
        w = np.where(a > 0, a * np.exp(-np.where(a > 0, z[i] - zmin, 0.0) / max(tau, 1e-6)), 0.0)
        csum += w[..., None] * np.where(w > 0, 1.0, 0.0)[..., None] * np.nan_to_num(col[i].astype(np.float64))
        wsum += w
    rgb = np.where((wsum > 1e-8)[..., None], csum / np.maximum(wsum, 1e-8)[..., None], bg)
    cover = (1.0 - rest)[..., None]
    return np.clip(rgb * cover + np.asarray(bg) * (1.0 - cover), 0.0, 1.0)


@pytest.mark.parametrize("n,depths,tau,thin", [
    (1, (1.0, 1.0), 0.1, 1.0), (33, (1.0, 1.2), 0.05, 1.0),             # a batch of 32 and one more
    (400, (1.0, 1.5), 0.05, 20.0),                                       # thin splats across the parts' corners
    (400, (1.0, 6.9), 0.1, 3.0), (400, (1.0, 7.1), 0.1, 3.0),            # depth ranges of 59 and 61 tau
    (400, (0.5, 60.0), 0.01, 1.0), (200, (1.0, 1.1), 1e-9, 1.0),         # far beyond
    (400, (1.0, 3.0), 1e4, 1.0)])                                        # all weights alike
def test_image_matches_float64(n, depths, tau, thin):
    """Ragged parts and tiles, every depth range, against the float64 image.
    The renderer's image bound, 1e-4."""
    rng = np.random.default_rng(n + int(thin))
    W, H, f, r_max = 50, 37, 40.0, 10
    z = rng.uniform(*depths, n)
    z[0], z[-1] = depths[0], depths[1]
    xy = (rng.uniform(-0.05, 1.05, (n, 2)) * [W, H] - [0.5 * W, 0.5 * H]) / f * z[:, None]
    R = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    size = (z / f)[:, None] * rng.uniform(0.4, 2.0, (n, 1)) * np.array([1.0, 1.0 / thin, 1.0 / thin])
    cov = (R * size[:, None, :] ** 2) @ R.transpose(0, 2, 1)
    xyz, cov, col = (a.astype(np.float32) for a in (np.c_[xy, z], cov, rng.uniform(0, 1, (n, 3))))
    t = lambda a: torch.tensor(a, device="cuda:0")
    cam = Camera(R=np.eye(3), T=np.zeros(3), fx=f, fy=f, width=W, height=H, device="cuda:0")
    bg = (0.1, 0.2, 0.3)
    img = render_gaussians(cam, t(xyz), t(cov), t(col), t(np.ones(n, np.float32)), bg=bg, r_max=r_max, tau=tau)
    want = _image64(xyz, cov, col, f, W, H, float(np.float32(tau)), bg, r_max)
    assert np.abs(img.cpu().numpy() - want).max() < 1e-4


def test_a_colour_that_is_not_finite_stays_in_its_footprint():
    """Infinite and NaN colours reach the pixels of their own footprint, no other of the same part."""
    f, W, H = 40.0, 32, 32
    u = np.array([4.5, 20.5, 27.5, 3.5])
    z = np.ones(4)
    xyz = np.c_[(u - 0.5 * W) / f, np.full(4, (6.5 - 0.5 * H) / f), z].astype(np.float32)
    cov = np.tile(np.eye(3, dtype=np.float32) * np.float32((0.1 / f) ** 2), (4, 1, 1))
    col = np.full((4, 3), 0.5, np.float32)
    bad = col.copy()
    bad[0], bad[2] = np.inf, np.nan
    t = lambda a: torch.tensor(a, device="cuda:0")
    cam = Camera(R=np.eye(3), T=np.zeros(3), fx=f, fy=f, width=W, height=H, device="cuda:0")
    a, b = (render_gaussians(cam, t(xyz), t(cov), t(c), t(np.ones(4, np.float32)), bg=(0, 0, 0), tau=0.1).cpu().numpy()
            for c in (col, bad))
    far = np.ones((H, W), bool)                       # radius 2 at most: ceil(3 sqrt(0.31))
    far[4:9, 2:7] = far[4:9, 25:30] = False
    assert np.isfinite(b[far]).all() and np.abs(a - b)[far].max() < 1e-6 and (b[far] > 0.1).any()
