"""Timed cases of the AnisoMPM framework, through its public entry points.

Each case is one call (or one short sequence of calls) that a simulation
program makes over and over: a substep, a frame of substeps, a frame of many
scenes, a differentiable rollout with its gradients, a rendered frame.  The
bodies are jittered particle lattices in the middle of a deformation: smooth
random displacement and velocity fields, the deformation gradient and APIC
matrix that belong to them, and partly damaged material, so that the
eigensolves, the damage drive and the stress split all have real work.

``exact`` restates the same steps in float64 with plain torch.
"""
import math

import torch

# ------------------------------------------------------------------------ the cases


def listed():
    return [
        # the smallest call: one eager substep of a 1,024-particle bar, as an interactive or
        # scripted loop issues it (host cost and launches count)
        dict(name="step_bar_1k", kind="step", n_grid=32, cx=8, cy=4, cz=4, ppc=2, dt=1e-4, shuffled=False),
        # the small benchmark bar (64^3 grid, 32x8x8 cells), a frame of 20 substeps
        dict(name="frame_bar_16k", kind="frame", n_grid=64, cx=32, cy=8, cz=8, ppc=2, dt=1e-4, n_sub=20,
             body="pulled", shuffled=False),
        # a block falling on colliders with every knob on (strain limit, damping, damage every
        # second substep); ragged particle count in no spatial order, as points sampled from a mesh
        dict(name="frame_drop_59k", kind="frame", n_grid=56, cx=23, cy=17, cz=19, ppc=2, dt=1e-4, n_sub=4,
             body="drop", shuffled=True),
        # the peel slab at 1/8 of its in-plane size with the directional interface law and the
        # per-frame observables of the experiment loop
        dict(name="frame_interface_138k", kind="frame", n_grid=256, cx=16, cy=20, cz=16, ppc=3, dt=2e-5, n_sub=6,
             body="interface", shuffled=False),
        # the headline: the 1,048,576-particle slab on 128^3
        dict(name="frame_slab_1m", kind="frame", n_grid=128, cx=64, cy=32, cz=64, ppc=2, dt=5e-5, n_sub=10,
             body="pulled", shuffled=False),
        # the largest single scene: the 8,847,360-particle peel slab on 256^3, 27 per cell, gravity
        dict(name="frame_peel_8m", kind="frame", n_grid=256, cx=128, cy=20, cz=128, ppc=3, dt=2e-5, n_sub=2,
             body="peel", shuffled=False),
        # a small batch of small uneven scenes (a parameter sweep)
        dict(name="batch_12_small", kind="batch", scenes=12, n_lo=4096, n_hi=16384, n_sub=4, dt=5e-5),
        # the batched workload: 64 uneven scenes, 4k to 256k particles, grids 32^3 to 128^3
        dict(name="batch_64", kind="batch", scenes=64, n_lo=4096, n_hi=262144, n_sub=4, dt=5e-5),
        # gradients of the small bar while part of it damages: forward, checkpoints and backward
        dict(name="grad_bar_16k", kind="grad", n_grid=64, cx=32, cy=8, cz=8, ppc=2, dt=1e-4, n_sub=12, every=4,
             shuffled=False),
        # gradients of the 1M slab
        dict(name="grad_slab_1m", kind="grad", n_grid=128, cx=64, cy=32, cz=64, ppc=2, dt=5e-5, n_sub=8, every=4,
             shuffled=False),
        # carrying and drawing one gaussian per particle of a 262,144-particle slab
        dict(name="render_262k", kind="render", n_grid=128, cx=32, cy=32, cz=32, ppc=2, width=1280, height=720),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, cells):
    """A box of about ``cells`` cells with a random aspect."""
    asp = [math.exp(rng.uniform(-0.6, 0.6)) for _ in range(3)]
    unit = (cells / (asp[0] * asp[1] * asp[2])) ** (1.0 / 3.0)
    return [max(3, int(round(unit * a))) for a in asp]


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "step", "batch", "grad", "render"])
    if kind == "batch":
        s = int(round(_log(rng, 2, 64)))
        lo = int(_log(rng, 1000, 8192))
        return dict(kind="batch", scenes=s, n_lo=lo, n_hi=int(lo * _log(rng, 2, 30)), n_sub=rng.choice([1, 2, 4]),
                    dt=5e-5)
    top = {"frame": 3.0e6, "step": 2.0e5, "grad": 6.0e5, "render": 2.5e5}[kind]
    ppc = 2 if kind == "render" else rng.choice([2, 2, 2, 3])
    c = _box(rng, _log(rng, 1000, top) / ppc ** 3)
    ng = int(min(256, max(24, math.ceil((rng.uniform(1.4, 2.5) * max(c) + 10) / 4.0) * 4 + rng.choice([0, 0, 1, 2]))))
    c = [min(v, ng - 10) for v in c]
    case = dict(kind=kind, n_grid=ng, cx=c[0], cy=c[1], cz=c[2], ppc=ppc)
    if kind == "render":
        return dict(case, width=rng.choice([640, 801, 960, 1280]), height=rng.choice([360, 480, 719, 720]))
    case.update(dt=rng.choice([2e-5, 5e-5]), shuffled=rng.random() < 0.25)
    if kind == "frame":
        case.update(n_sub=rng.choice([2, 3, 4, 5]), body=rng.choice(["pulled", "drop", "interface", "peel"]))
    if kind == "grad":
        case.update(n_sub=rng.choice([4, 6, 7]), every=rng.choice([2, 3, 4]))
    return case


# ------------------------------------------------------------------------ inputs


def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _body(n_grid, cells, ppc, seed, body, dt, shuffled, E0=1.0e4, nu=0.3, sigma0=200.0):
    """float32 inputs of one scene: particle state and material, boundary
    conditions and constants, made from the seed alone."""
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    f64 = dict(device=dev, dtype=torch.float64)
    rand = lambda *s: torch.rand(*s, generator=g, **f64)
    randn = lambda *s: torch.randn(*s, generator=g, **f64)
    dx = 1.0 / n_grid
    lo = [(n_grid - c) // 2 for c in cells]
    if body == "drop":
        lo[1] = 7
    ax = [torch.arange(c, **f64) + l for c, l in zip(cells, lo)]
    cell = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 1, 3)
    sub = (torch.arange(ppc, **f64) + 0.5) / ppc
    sub = torch.stack(torch.meshgrid(sub, sub, sub, indexing="ij"), -1).reshape(1, -1, 3)
    x = ((cell + sub) * dx).reshape(-1, 3)
    n = x.shape[0]
    x = x + (2.0 * rand(n, 3) - 1.0) * (0.5 / ppc * dx * 0.5)
    if shuffled:   # sampled points: no spatial order, and a few of them left out
        x = x[torch.randperm(n, generator=g, device=dev)][: n - n % 7 - 1]
        n = x.shape[0]
    blo = torch.tensor([l * dx for l in lo], **f64)
    ext = torch.tensor([c * dx for c in cells], **f64)
    xi = (x - blo) / ext
    eye = torch.eye(3, **f64)

    def field(modes, amp):   # a smooth vector field with gradients of size amp, and its gradient
        u, G = torch.zeros(n, 3, **f64), torch.zeros(n, 3, 3, **f64)
        for _ in range(modes):
            k = 2.0 * math.pi * (2.0 * rand(3) - 1.0) * 0.8
            c = randn(3) / math.sqrt(modes)
            ph = xi @ k + 6.28 * rand(1)
            kk = k / ext
            s = amp / (kk.norm() + 1e-9)
            u = u + s * torch.sin(ph)[:, None] * c
            G = G + s * torch.cos(ph)[:, None, None] * (c[:, None] * kk[None, :])
        return u, G

    u, Gu = field(3, 0.02)
    shift = 0.4 * dx / max(float(u.abs().max()), 0.4 * dx)   # displaced by less than half a cell
    F = eye + Gu + 2e-3 * randn(n, 3, 3)
    v, Gv = field(3, 6.0)
    vs = 0.5 / max(float(v.abs().max()), 0.5)
    v, Gv = v * vs, Gv * vs
    hurt = torch.sigmoid(12.0 * (torch.cos(4.0 * xi[:, 0] + 2.0 * xi[:, 2] + 6.28 * rand(1)) - 0.7))
    d = (0.05 * rand(n) + 0.5 * hurt * rand(n)).clamp(0.0, 0.95)
    D_hist = (0.5 + 2.5 * hurt) * rand(n)
    lap = 0.02 / dx ** 2 * randn(n)
    if body == "loaded":
        # one part of the body stretched well past its critical stress and damaging, the rest well
        # below it: away from the drive's thresholds the gradients are smooth functions of the inputs
        part = (torch.sin(5.0 * xi[:, 0] + 3.0 * xi[:, 1]) > 0.3).double()
        stretch = torch.tensor([1.5, 1.0, 0.5], **f64) * eye
        F = eye + (0.005 + 0.02 * part)[:, None, None] * stretch + 0.02 * Gu + 2e-4 * randn(n, 3, 3)
        d = 0.02 + 0.03 * rand(n)
        D_hist = 0.5 + 0.5 * rand(n)
        lap = 0.1 * lap
        rise = (0.3 * xi[:, 1] ** 2).clamp(0.0, 0.3)   # at rest at the held layer
        v, Gv = v * rise[:, None], Gv * rise[:, None, None]
    E = E0 * torch.exp((0.05 if body == "loaded" else 0.2) * randn(n))
    fib = torch.tensor([1.0, 0.0, 0.0], **f64) + 0.25 * randn(n, 3)
    fib = fib / fib.norm(dim=1, keepdim=True)
    f32 = lambda t: t.to(torch.float32).contiguous()
    out = dict(x=f32(x + shift * u), v=f32(v), F=f32(F), C=f32(Gv), d=f32(d), lap=f32(lap),
               D_hist=f32(D_hist), vol=f32(torch.full((n,), (dx / ppc) ** 3, **f64)), E=f32(E), fib=f32(fib),
               sigma_c=f32((2.0 if body == "loaded" else 1.0) * sigma0 * (0.9 + 0.2 * rand(n))))
    out["mu"] = out["E"] / (2.0 * (1.0 + nu))
    out["lam"] = out["E"] * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))
    a = out["fib"] / (out["fib"].norm(dim=1, keepdim=True) + 1e-12)
    out["A0"] = eye.to(torch.float32) - a[:, :, None] * a[:, None, :]
    bottom = xi[:, 1] * cells[1] < 1.0
    top = (xi[:, 1] * cells[1] > cells[1] - 1.0) & (xi[:, 0] * cells[0] < 1.0)
    prm = dict(n_grid=n_grid, dx=dx, dt=dt, rho=1000.0, nu=nu, l0_scale=1.0, eta=1e-3, zeta=1.0, residual=1e-3,
               gravity=(0.0, 0.0, 0.0), grid_damp=1.0, f_clamp=None, damage_every=1, grips=[], colliders=[],
               interface=None, groups=None)
    if body == "clamped":   # both ends held: the bar swings, however often it is stepped
        ends = (xi[:, 0] * cells[0] < 1.0) | (xi[:, 0] * cells[0] > cells[0] - 1.0)
        prm["grips"] = [(ends, (0.0, 0.0, 0.0), 0.0)]
        out["allow"] = ~ends
    elif body in ("held", "loaded"):   # standing on a clamped bottom layer and swinging
        prm["grips"] = [(bottom, (0.0, 0.0, 0.0), 0.0)]
        out["allow"] = ~bottom
    elif body == "drop":
        prm.update(gravity=(0.0, -9.8, 0.0), grid_damp=0.999, f_clamp=(0.9, 1.1), damage_every=2, zeta=1.3,
                   l0_scale=0.7, eta=5e-3, residual=5e-3)
        ctr = [(l + 0.5 * c) * dx for l, c in zip(lo, cells)]
        prm["colliders"] = [
            ("halfspace", (0.0, 8.43 * dx, 0.0), (0.0, 0.0, 0.0), (0.1, 1.0, 0.0), 0.0, "slip", 0.4),
            ("sphere", (lo[0] * dx, ctr[1], ctr[2]), (3.0, 0.0, 0.0), None, 2.53 * dx, "sticky", 0.0),
            ("sphere", (ctr[0], (lo[1] + cells[1]) * dx, ctr[2]), (0.0, -2.0, 0.0), None, 2.07 * dx, "slip", 0.2)]
        out["allow"] = torch.ones(n, dtype=torch.bool, device=dev)
    else:
        prm["grips"] = [(bottom, (0.0, 0.0, 0.0), 0.0),
                        (top, (0.0, 1.0, 0.2), 1e-3 if body == "interface" else 0.0)]
        out["allow"] = ~(bottom | top)
        if body == "peel":
            prm["gravity"] = (0.0, -9.8, 0.0)
            bond = (xi[:, 1] > 0.7) & (xi[:, 1] < 0.76)
            out["sigma_c"] = torch.where(bond, 0.2 * out["sigma_c"], 2.0 * out["sigma_c"])
        if body == "interface":
            band = (xi[:, 1] - 0.6).abs() < 0.12
            nrm = torch.tensor([0.0, 1.0, 0.0], **f64) + 0.05 * randn(n, 3)
            nrm = f32(nrm)
            out["normals"] = nrm / (nrm.norm(dim=1, keepdim=True) + 1e-12)
            out["band"] = band
            nn = out["normals"][:, :, None] * out["normals"][:, None, :]
            out["A0"] = torch.where(band[:, None, None], nn, out["A0"])
            out["sigma_c"] = torch.where(band, 0.3 * out["sigma_c"], out["sigma_c"])
            prm["interface"] = True
            prm["groups"] = dict(interface=band, flesh=~band & (xi[:, 1] < 0.6), peel=~band & (xi[:, 1] >= 0.6))
    out["mass"] = out["vol"] * prm["rho"]
    return out, prm


def _cells(case):
    return [case["cx"], case["cy"], case["cz"]]


def _inputs(case, seed):
    """[(inputs, constants)] of the case's scenes."""
    if case["kind"] != "batch":
        body = {"step": "clamped", "grad": "loaded", "render": "pulled"}.get(case["kind"], case.get("body"))
        return [_body(case["n_grid"], _cells(case), case["ppc"], seed, body, case.get("dt", 5e-5),
                      case.get("shuffled", False))]
    g = torch.Generator().manual_seed(12345)   # the scenes' sizes belong to the case, not to the seed
    out = []
    for k in range(case["scenes"]):
        r = torch.rand(6, generator=g, dtype=torch.float64).tolist()
        cells = max(8.0, math.exp(math.log(case["n_lo"]) + r[0] * math.log(case["n_hi"] / case["n_lo"])) / 8.0)
        asp = [math.exp(r[1] - 0.5), 0.5 * math.exp(r[2] - 0.5), math.exp(r[3] - 0.5)]
        unit = (cells / (asp[0] * asp[1] * asp[2])) ** (1.0 / 3.0)
        ext = [max(2, int(round(unit * a))) for a in asp]
        ng = int(min(128, max(32, math.ceil((2.0 * max(ext) + 8) / 16.0) * 16)))
        out.append(_body(ng, ext, 2, seed * 1009 + k, "held", case["dt"], False, E0=1e3 * 10 ** (2 * r[4]),
                         nu=0.2 + 0.25 * r[5], sigma0=50.0 + 300.0 * r[4]))
    return out


# ------------------------------------------------------------------------ the framework's side

STATE = ("x", "v", "F", "C", "d", "lap", "D_hist")


def _solver(inp, prm):
    import peel_mpm_b200 as pm
    sim = pm.AnisoMPM(n_grid=prm["n_grid"], grid_lim=1.0, dt=prm["dt"], gravity=prm["gravity"],
                      grid_damp=prm["grid_damp"], f_clamp=prm["f_clamp"], damage_every=prm["damage_every"],
                      device="cuda:0")
    sim.add_object(inp["x"], inp["vol"], rho=prm["rho"], E=1e4, nu=prm["nu"], fibers=inp["fib"], alpha=-1.0,
                   l0_scale=prm["l0_scale"], eta=prm["eta"], zeta=prm["zeta"], residual=prm["residual"])
    for f in STATE[1:] + ("mu", "lam", "sigma_c", "A0"):
        setattr(sim, f, inp[f])
    sim.allow = inp["allow"]
    if prm["interface"]:
        sim.n_interface = torch.where(inp["band"][:, None], inp["normals"], torch.zeros_like(inp["normals"]))
        sim.interface_mask = inp["band"]
    for mask, vel, ramp in prm["grips"]:
        sim.particle_bc.append(pm.grip_bc(mask, vel, ramp))
    for kind, o, w, nrm, rad, mode, fr in prm["colliders"]:
        fn = lambda t, o=o, w=w: [o[0] + w[0] * t, o[1] + w[1] * t, o[2] + w[2] * t]
        sim.colliders.append(pm.halfspace_collider(fn, nrm, mode=mode, friction=fr) if kind == "halfspace"
                             else pm.sphere_collider(fn, rad, mode=mode, friction=fr))
    return sim


def _camera(case, seed):
    """Camera constants of a view of the slab from above and aside."""
    az, el = 0.6 + 0.05 * (seed % 7), 0.5
    fwd = [-math.cos(el) * math.sin(az), -math.sin(el), -math.cos(el) * math.cos(az)]
    right = [math.cos(az), 0.0, -math.sin(az)]
    down = [fwd[1] * right[2] - fwd[2] * right[1], fwd[2] * right[0] - fwd[0] * right[2],
            fwd[0] * right[1] - fwd[1] * right[0]]
    R = [[right[i], down[i], fwd[i]] for i in range(3)]
    size = max(case["cx"], case["cy"], case["cz"]) / case["n_grid"]
    dist = 2.2 * size
    T = [-sum(0.5 * R[i][j] for i in range(3)) + (dist if j == 2 else 0.0) for j in range(3)]
    return R, T, 0.9 * case["width"]


def _splats(case, seed, n):
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed) + 77)
    dx = 1.0 / case["n_grid"]
    off = 0.1 * dx * torch.randn(n, 3, generator=g, device=dev)
    L = 0.12 * dx * (torch.eye(3, device=dev) + 0.3 * torch.randn(n, 3, 3, generator=g, device=dev))
    cov = L @ L.transpose(1, 2)
    col = torch.rand(n, 3, generator=g, device=dev)
    return off, cov, col, torch.ones(n, device=dev)


def prepare(case, seed):
    scenes = _inputs(case, seed)
    sims = [_solver(i, p) for i, p in scenes]
    st = dict(case=case, sims=sims, sim=sims[0], start=[{f: i[f] for f in STATE} for i, _ in scenes])
    kind = case["kind"]
    if kind == "batch":
        import peel_mpm_b200 as pm
        st["batch"] = pm.BatchedAnisoMPM(sims)
    elif kind == "grad":
        inp, prm = scenes[0]
        st["par"] = {k: inp[k].clone().requires_grad_(True) for k in ("E", "fib", "sigma_c", "v")}
        st["wx"], st["wv"] = _weights(inp)
        st["nu"] = prm["nu"]
    elif kind == "render":
        from peel_mpm_b200.render import Camera, world_map
        import numpy as np
        R, T, f = _camera(case, seed)
        st["cam"] = Camera(R=np.array(R), T=np.array(T), fx=f, fy=f, width=case["width"], height=case["height"])
        n = sims[0].n
        st["splats"] = _splats(case, seed, n)
        st["bind"] = torch.arange(n, dtype=torch.int32, device="cuda:0")
        st["map"] = world_map()
    if scenes[0][1]["groups"] is not None:
        from peel_mpm_b200.observables import FrameObservables
        st["obs"] = FrameObservables(sims[0], scenes[0][1]["groups"], max_frames=4)
    return st


def _reset(sim, start):
    for f in STATE:
        getattr(sim, f).copy_(start[f])


def _state(sim):
    return {f: getattr(sim, f) for f in STATE}


def _weights(inp):
    """Smooth weights of the loss on final positions and velocities."""
    x = inp["x"]
    wx = torch.sin(9.0 * x + torch.tensor([0.3, 1.1, 2.0], device=x.device))
    wv = torch.cos(7.0 * x.flip(1) + torch.tensor([1.3, 0.1, 0.7], device=x.device))
    return wx / x.shape[0], 0.01 * wv / x.shape[0]


def run(st):
    case, sim = st["case"], st["sim"]
    kind = case["kind"]
    if kind == "step":
        sim.substep(0.0)
        return _state(sim)
    if kind == "frame":
        _reset(sim, st["start"][0])   # every pass runs the same frame
        sim.run_frame(case["n_sub"], 0.0)
        out = _state(sim)
        if "obs" in st:
            st["obs"].update(0)
            out.update(phi=sim.phi, phi_shear=sim.phi_shear, table=st["obs"].table[0])
        return out
    if kind == "batch":
        st["batch"].run_frame(case["n_sub"], 0.0)
        # a field of every scene, each field of some scenes
        return [getattr(s, STATE[k % len(STATE)]) for k, s in enumerate(st["sims"])]
    if kind == "grad":
        from peel_mpm_b200 import differentiable as dfx
        _reset(sim, st["start"][0])
        p = st["par"]
        mu, lam, A0 = dfx.material(p["E"], st["nu"], p["fib"], -1.0)
        x, v = dfx.rollout(sim, case["n_sub"], mu=mu, lam=lam, sigma_c=p["sigma_c"], A0=A0, v0=p["v"],
                           checkpoint_every=case["every"], outputs="xv")
        loss = (st["wx"] * x).sum() + (st["wv"] * v).sum()
        gr = torch.autograd.grad(loss, [p[k] for k in ("E", "fib", "sigma_c", "v")])
        return {"x": x.detach(), "v": v.detach(), "E": gr[0], "fib": gr[1], "sigma_c": gr[2], "v0": gr[3]}
    from peel_mpm_b200.render import carry_gaussians, render_gaussians
    off, cov, col, op = st["splats"]
    pos, cw, cc = carry_gaussians(sim, st["bind"], off, cov, col, sim_to_world=st["map"], crack_tint=0.6,
                                  check_bind=False)
    return {"pos": pos, "cov": cw, "color": cc, "image": render_gaussians(st["cam"], pos, cw, cc, op)}


# ------------------------------------------------------------------------ floor

_MUTABLE, _FIXED, _NODE = 108, 73, 80   # bytes: state read and written, material read, per active node


def _count(cells, ppc):
    """Particles and active nodes of a box."""
    n = cells[0] * cells[1] * cells[2] * ppc ** 3
    return n, (cells[0] + 5) * (cells[1] + 5) * (cells[2] + 5)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        boxes, g = [], torch.Generator().manual_seed(12345)
        for _ in range(case["scenes"]):
            r = torch.rand(6, generator=g, dtype=torch.float64).tolist()
            c = max(8.0, math.exp(math.log(case["n_lo"]) + r[0] * math.log(case["n_hi"] / case["n_lo"])) / 8.0)
            a = [math.exp(r[1] - 0.5), 0.5 * math.exp(r[2] - 0.5), math.exp(r[3] - 0.5)]
            u = (c / (a[0] * a[1] * a[2])) ** (1.0 / 3.0)
            boxes.append(_count([max(2, int(round(u * v))) for v in a], 2))
        n, nodes = sum(b[0] for b in boxes), sum(b[1] for b in boxes)
    else:
        n, nodes = _count(_cells(case), case["ppc"])
    if kind == "render":   # carried gaussians (read 176 B, write 60), splats read again, the image written
        return {"bytes": n * (176.0 + 2 * 60.0) + 12.0 * case["width"] * case["height"], "flops": n * 400.0}
    step = n * (2.0 * _MUTABLE + _FIXED) + nodes * _NODE
    flops = n * 2500.0
    subs = case.get("n_sub", 1)
    if kind == "grad":
        # forward once, then per substep the adjoint reads the states before and after, the material and
        # the state's adjoint and writes the adjoint; parameter gradients are written once
        back = n * (2.0 * _MUTABLE + _FIXED + 2.0 * _MUTABLE) + 2.0 * nodes * _NODE
        return {"bytes": subs * (step + back) + 48.0 * n, "flops": subs * n * 8000.0}
    return {"bytes": subs * step, "flops": subs * flops}


# ------------------------------------------------------------------------ the same steps in float64


def _jacobi(A):
    """Eigenvalues (n,3) and eigenvectors (n,3,3) of symmetric float64 matrices by cyclic Jacobi rotations."""
    a = [[A[:, i, j].clone() for j in range(3)] for i in range(3)]
    one, zero = torch.ones_like(a[0][0]), torch.zeros_like(a[0][0])
    V = [[(one if i == j else zero).clone() for j in range(3)] for i in range(3)]
    for _ in range(8):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            r = 3 - p - q
            apq = a[p][q]
            th = (a[q][q] - a[p][p]) / torch.where(apq.abs() > 1e-300, 2.0 * apq, one)
            t = torch.where(th >= 0, one, -one) / (th.abs() + torch.sqrt(th * th + 1.0))
            t = torch.where(apq.abs() > 1e-300, t, zero)
            c = 1.0 / torch.sqrt(t * t + 1.0)
            s = t * c
            app, aqq, apr, aqr = a[p][p], a[q][q], a[p][r], a[q][r]
            a[p][p], a[q][q] = app - t * apq, aqq + t * apq
            a[p][q] = a[q][p] = zero
            a[p][r] = a[r][p] = c * apr - s * aqr
            a[q][r] = a[r][q] = s * apr + c * aqr
            for i in range(3):
                vp, vq = V[i][p], V[i][q]
                V[i][p], V[i][q] = c * vp - s * vq, s * vp + c * vq
    return torch.stack([a[i][i] for i in range(3)], 1), torch.stack([torch.stack(r, 1) for r in V], 1)


class _Positive(torch.autograd.Function):
    """Positive part of a symmetric matrix, with the divided-difference derivative of a spectral function."""

    @staticmethod
    def forward(ctx, A):
        e, Q = _jacobi(A)
        ctx.save_for_backward(e, Q)
        return (Q * e.clamp(min=0.0)[:, None, :]) @ Q.transpose(1, 2)

    @staticmethod
    def backward(ctx, g):
        e, Q = ctx.saved_tensors
        B = Q.transpose(1, 2) @ (0.5 * (g + g.transpose(1, 2))) @ Q
        ei, ej = e[:, :, None], e[:, None, :]
        de = ei - ej
        same = de.abs() <= 1e-12 * (ei.abs() + ej.abs())
        pos = (e >= 0).to(e.dtype)
        G = torch.where(same, 0.5 * (pos[:, :, None] + pos[:, None, :]),
                        (ei.clamp(min=0) - ej.clamp(min=0)) / torch.where(same, torch.ones_like(de), de))
        return Q @ (G * B) @ Q.transpose(1, 2)


def _polar(F):
    """Rotation of the polar decomposition (det F > 0) by Newton's iteration R <- (R + R^-T) / 2."""
    R = F
    for _ in range(9):
        c = torch.stack([torch.linalg.cross(R[:, 1], R[:, 2]), torch.linalg.cross(R[:, 2], R[:, 0]),
                         torch.linalg.cross(R[:, 0], R[:, 1])], 1)   # cofactors = det R^-T
        det = (R[:, 0] * c[:, 0]).sum(1)
        R = 0.5 * (R + c / det[:, None, None])
    return R


def _dot3(a, b):
    return (a * b).sum(-1)


def _resolve64(v, vc, nn, mode, fr):
    if mode == "sticky":
        return vc.expand_as(v)
    r = v - vc
    vn = _dot3(r, nn)
    inward = vn.clamp(max=0.0)
    t = r - vn[:, None] * nn
    if fr > 0:
        sc = 1.0 + fr * inward / (t.norm(dim=1) + 1e-9)
        t = t * sc.clamp(min=0.0)[:, None]
    return vc + t + (vn - inward)[:, None] * nn


def _step64(S, M, prm, t, step):
    """One substep of the state dict S with material M (all float64)."""
    ng, dx, dt = prm["n_grid"], prm["dx"], prm["dt"]
    inv = 1.0 / dx
    x, v, F, C = S["x"], S["v"], S["F"], S["C"]
    n, dev = x.shape[0], x.device
    for mask, vel, ramp in prm["grips"]:
        f = min(t / ramp, 1.0) if ramp > 0 else 1.0
        v = torch.where(mask[:, None], torch.tensor([c * f for c in vel], dtype=x.dtype, device=dev), v)
    I = torch.eye(3, dtype=x.dtype, device=dev)
    R = _polar(F)
    if prm["f_clamp"] is not None:
        lam_, V = _jacobi(F.transpose(1, 2) @ F)
        sv = lam_.clamp(min=1e-12).sqrt()
        sc = sv.clamp(*prm["f_clamp"])
        F = F @ ((V * (sc / sv.clamp(min=1e-12))[:, None, :]) @ V.transpose(1, 2))
        J = sc.prod(1).clamp(min=1e-6)
    else:
        J = (F[:, 0] * torch.linalg.cross(F[:, 1], F[:, 2])).sum(1).clamp(min=1e-6)
    tdev = 2.0 * M["mu"][:, None, None] * ((F - R) @ F.transpose(1, 2))
    tv = M["lam"] * (J - 1.0) * J
    tau0 = tdev + tv[:, None, None] * I
    d, Dh = S["d"], S["D_hist"]
    phi = phs = None
    if bool(M["allow"].any()) and step % prm["damage_every"] == 0:
        sig = tau0 / J[:, None, None]
        sp = _Positive.apply(0.5 * (sig + sig.transpose(1, 2)))
        A = R @ M["A0"] @ R.transpose(1, 2)
        MM = A @ sp
        phi = (MM * MM.transpose(1, 2)).sum((1, 2)) / M["sigma_c"] ** 2
        if prm["interface"]:
            nn = M["n0"]
            s = (sp @ nn[:, :, None])[:, :, 0]
            tt = s - _dot3(s, nn)[:, None] * nn
            phs = _dot3(tt, tt) / M["sigma_c"] ** 2
        Dh = torch.maximum(Dh, prm["zeta"] * (phi - 1.0).clamp(min=0.0))
        l0 = prm["l0_scale"] * dx
        dd = ((1.0 - d) * Dh - (d - l0 * l0 * S["lap"])).clamp(min=0.0)
        dn = (d + dt * prm["damage_every"] / prm["eta"] * dd).clamp(0.0, 1.0)
        d = torch.where(M["allow"], torch.maximum(dn, d), d)
    g = (1.0 - d) ** 2 * (1.0 - prm["residual"]) + prm["residual"]
    vdeg = torch.where(J >= 1.0, g, torch.ones_like(g))
    tau = g[:, None, None] * tdev + (vdeg * tv)[:, None, None] * I
    if prm["interface"]:
        m = (F @ M["n0"][:, :, None])[:, :, 0]
        m = m / (m.norm(dim=1, keepdim=True) + 1e-9)
        P = m[:, :, None] * m[:, None, :]
        Q = I - P
        gI = torch.where((m[:, None, :] @ tau0 @ m[:, :, None])[:, 0, 0] > 0, g, torch.ones_like(g))[:, None, None]
        gg = g[:, None, None]
        td = Q @ tau0 @ Q + gI * (P @ tau0 @ P) + gg * (P @ tau0 @ Q + Q @ tau0 @ P)
        tau = torch.where(M["band"][:, None, None], td, tau)
    aff = (-dt * M["vol"] * 4.0 * inv * inv)[:, None, None] * tau + M["mass"][:, None, None] * C
    X = x * inv
    qb = torch.floor(X - 0.5)
    fx = X - qb
    qw = [0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1.0) ** 2, 0.5 * (fx - 0.5) ** 2]
    cb = torch.floor(X)
    f = X - cb
    o1 = 1.0 - f
    cw = [o1 ** 3 / 6.0, 2.0 / 3.0 - f * f + 0.5 * f ** 3, 2.0 / 3.0 - o1 * o1 + 0.5 * o1 ** 3, f ** 3 / 6.0]
    c2 = [o1, 3.0 * f - 2.0, 1.0 - 3.0 * f, f]
    qi, ci = qb.long(), cb.long() - 1
    at = lambda b, o: ((b[:, 0] + o[0]).clamp(0, ng - 1) * ng + (b[:, 1] + o[1]).clamp(0, ng - 1)) * ng + \
        (b[:, 2] + o[2]).clamp(0, ng - 1)
    q27 = [(i, j, k) for i in range(3) for j in range(3) for k in range(3)]
    c64 = [(i, j, k) for i in range(4) for j in range(4) for k in range(4)]
    off = lambda o: (torch.tensor(o, dtype=x.dtype, device=dev) - fx) * dx
    gm = torch.zeros(ng ** 3, dtype=x.dtype, device=dev)
    gmv = torch.zeros(ng ** 3, 3, dtype=x.dtype, device=dev)
    mv = M["mass"][:, None] * v
    for o in q27:
        w = qw[o[0]][:, 0] * qw[o[1]][:, 1] * qw[o[2]][:, 2]
        idx = at(qi, o)
        gmv = gmv.index_add(0, idx, w[:, None] * (mv + (aff @ off(o)[:, :, None])[:, :, 0])) if x.requires_grad or \
            v.requires_grad or aff.requires_grad else gmv.index_add_(0, idx, w[:, None] *
                                                                     (mv + (aff @ off(o)[:, :, None])[:, :, 0]))
        gm = gm.index_add(0, idx, w * M["mass"]) if w.requires_grad else gm.index_add_(0, idx, w * M["mass"])
    gd = torch.zeros_like(gm)
    gw = torch.zeros_like(gm)
    for o in c64:
        w = cw[o[0]][:, 0] * cw[o[1]][:, 1] * cw[o[2]][:, 2]
        idx = at(ci, o)
        gd = gd.index_add(0, idx, w * d) if (w.requires_grad or d.requires_grad) else gd.index_add_(0, idx, w * d)
        gw = gw.index_add(0, idx, w) if w.requires_grad else gw.index_add_(0, idx, w)
    live = gm > 1e-12
    gv = gmv / torch.where(live, gm, torch.ones_like(gm))[:, None]
    gv = (gv + dt * torch.tensor(prm["gravity"], dtype=x.dtype, device=dev)) * prm["grid_damp"]
    gv = torch.where(live[:, None], gv, torch.zeros_like(gv))
    if prm["colliders"]:
        ids = torch.arange(ng ** 3, device=dev)
        pos = torch.stack([ids // (ng * ng), ids // ng % ng, ids % ng], 1).to(x.dtype) * dx
        for kind, o, w, nrm, rad, mode, fr in prm["colliders"]:
            c = torch.tensor([a + b * t for a, b in zip(o, w)], dtype=x.dtype, device=dev)
            vc = torch.tensor(w, dtype=x.dtype, device=dev)
            r = pos - c
            if kind == "halfspace":
                nn = torch.tensor(nrm, dtype=x.dtype, device=dev)
                nn = (nn / nn.norm()).expand_as(r)
                hit = _dot3(r, nn) < 0
            else:
                ds = r.norm(dim=1)
                hit, nn = ds < rad, r / (ds + 1e-9)[:, None]
            gv = torch.where((hit & live)[:, None], _resolve64(gv, vc, nn, mode, fr), gv)
    wl = gw > 1e-12
    gd = torch.where(wl, gd / torch.where(wl, gw, torch.ones_like(gw)), torch.zeros_like(gd))
    nv, nC, lap = torch.zeros_like(x), torch.zeros_like(C), torch.zeros_like(d)
    for o in q27:
        w = qw[o[0]][:, 0] * qw[o[1]][:, 1] * qw[o[2]][:, 2]
        gn = w[:, None] * gv[at(qi, o)]
        nv = nv + gn
        nC = nC + gn[:, :, None] * off(o)[:, None, :]
    for o in c64:
        a, b, c = o
        L = c2[a][:, 0] * cw[b][:, 1] * cw[c][:, 2] + cw[a][:, 0] * c2[b][:, 1] * cw[c][:, 2] + \
            cw[a][:, 0] * cw[b][:, 1] * c2[c][:, 2]
        lap = lap + L * gd[at(ci, o)]
    nC = nC * (4.0 * inv * inv)
    out = dict(x=(x + dt * nv).clamp(2.0 * dx, 1.0 - 2.0 * dx), v=nv, F=(I + dt * nC) @ F, C=nC, d=d,
               lap=lap * inv * inv, D_hist=Dh)
    return out, phi, phs


def _f64(inp):
    d = lambda t: t.double() if t.is_floating_point() else t
    S = {f: d(inp[f]) for f in STATE}
    M = {k: d(inp[k]) for k in ("mu", "lam", "sigma_c", "A0", "vol", "mass", "allow")}
    if "band" in inp:
        M["band"] = inp["band"]
        M["n0"] = torch.where(inp["band"][:, None], d(inp["normals"]), torch.zeros_like(d(inp["normals"])))
    return S, M


def _frame64(inp, prm, subs):
    S, M = _f64(inp)
    phi = phs = None
    for s in range(subs):
        S, p, q = _step64(S, M, prm, s * prm["dt"], s)
        phi, phs = (p, q) if p is not None else (phi, phs)
    return S, phi, phs


def exact(case, seed):
    kind = case["kind"]
    scenes = _inputs(case, seed)
    if kind == "render":
        return _render64(case, seed, scenes[0][0])
    if kind == "grad":
        return _grad64(case, *scenes[0])
    with torch.no_grad():
        got = [_frame64(i, p, case.get("n_sub", 1)) for i, p in scenes]
    if kind == "batch":
        return [g[0][STATE[k % len(STATE)]] for k, g in enumerate(got)]
    S, phi, phs = got[0]
    groups = scenes[0][1]["groups"]
    if groups is not None:
        row = []
        for m in groups.values():
            d = S["d"][m]
            row.append(torch.stack([phi[m].max(), phs[m].max(), d.sum(), d.max(), (d > 0.5).double().sum(),
                                    m.double().sum(), S["x"][m][:, 1].sum(), d.new_zeros(())]))
        S = dict(S, phi=phi, phi_shear=phs, table=torch.stack(row))
    return S


def _grad64(case, inp, prm):
    from torch.utils.checkpoint import checkpoint
    S, M = _f64(inp)
    E, fib, sc, v0 = (inp[k].double().requires_grad_(True) for k in ("E", "fib", "sigma_c", "v"))
    nu = prm["nu"]
    a = fib / (fib.norm(dim=1, keepdim=True) + 1e-12)
    mu, lam = E / (2.0 * (1.0 + nu)), E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))
    A0 = torch.eye(3, dtype=E.dtype, device=E.device) - a[:, :, None] * a[:, None, :]

    def one(s, mu, lam, sc, A0, *state):
        out, _, _ = _step64(dict(zip(STATE, state)), dict(M, mu=mu, lam=lam, sigma_c=sc, A0=A0), prm, s * prm["dt"], s)
        return tuple(out[f] for f in STATE)

    state = tuple(v0 if f == "v" else S[f] for f in STATE)
    for s in range(case["n_sub"]):
        state = checkpoint(one, s, mu, lam, sc, A0, *state, use_reentrant=False)
    wx, wv = (w.double() for w in _weights(inp))
    loss = (wx * state[0]).sum() + (wv * state[1]).sum()
    gE, gf, gs, gv = torch.autograd.grad(loss, [E, fib, sc, v0])
    return {"x": state[0].detach(), "v": state[1].detach(), "E": gE, "fib": gf, "sigma_c": gs, "v0": gv}


def _render64(case, seed, inp):
    """Carried gaussians, and their image: EWA projection and the soft depth buffer over each splat's square."""
    n = inp["x"].shape[0]
    off, cov, col, _ = (t.double() for t in _splats(case, seed, n))
    x, F, d = inp["x"].double(), inp["F"].double(), inp["d"].double()
    pos = x + (F @ off[:, :, None])[:, :, 0]
    cov = F @ cov @ F.transpose(1, 2)
    color = col * (1.0 - 0.6 * d)[:, None]
    R, T, fl = _camera(case, seed)
    R, T = torch.tensor(R, dtype=x.dtype, device=x.device), torch.tensor(T, dtype=x.dtype, device=x.device)
    W, H, r_max = case["width"], case["height"], 10
    Xc = pos @ R + T
    z = Xc[:, 2]
    ok = z > 0.05
    u, v = fl * Xc[:, 0] / z + W / 2.0, fl * Xc[:, 1] / z + H / 2.0
    Jm = torch.zeros(n, 2, 3, dtype=x.dtype, device=x.device)
    Jm[:, 0, 0] = Jm[:, 1, 1] = fl / z
    Jm[:, 0, 2], Jm[:, 1, 2] = -fl * Xc[:, 0] / z ** 2, -fl * Xc[:, 1] / z ** 2
    c2 = Jm @ (R.t() @ cov @ R) @ Jm.transpose(1, 2)
    a, b, c = c2[:, 0, 0] + 0.3, c2[:, 0, 1], c2[:, 1, 1] + 0.3
    det = a * c - b * b
    mid = 0.5 * (a + c)
    raw = 3.0 * (mid + (mid * mid - det).clamp(min=0).sqrt()).clamp(min=1e-6).sqrt()
    rad = raw.ceil().clamp(1, r_max)
    u0, v0 = u.floor(), v.floor()
    ok = ok & (det > 1e-9) & (raw < 70) & (u0 + rad >= 0) & (u0 - rad < W) & (v0 + rad >= 0) & (v0 - rad < H)
    i = ok.nonzero()[:, 0]
    u, v, u0, v0, z, rad, a, b, c, det = (t[i] for t in (u, v, u0, v0, z, rad, a, b, c, det))
    color_i = color[i]
    tau = max(0.02 * float(z.median()), 1e-6)
    zmin = torch.full((W * H,), float("inf"), dtype=x.dtype, device=x.device)
    acc = torch.zeros(W * H, 4, dtype=x.dtype, device=x.device)
    lg = torch.zeros(W * H, dtype=x.dtype, device=x.device)
    for phase in (0, 1):
        for oy in range(-r_max, r_max + 1):
            for ox in range(-r_max, r_max + 1):
                px, py = u0 + ox, v0 + oy
                k = (rad >= max(abs(ox), abs(oy))) & (px >= 0) & (px < W) & (py >= 0) & (py < H)
                dxp, dyp = px + 0.5 - u, py + 0.5 - v
                power = (-0.5 * (c * dxp * dxp + a * dyp * dyp) + b * dxp * dyp) / det
                al = torch.exp(power.clamp(max=0.0))
                k = k & (al > 1.0 / 255.0)
                at = torch.where(k, py * W + px, torch.zeros_like(px)).long()
                if phase == 0:
                    zmin.scatter_reduce_(0, at, torch.where(k, z, torch.full_like(z, float("inf"))), "amin")
                else:
                    w = torch.where(k, al * torch.exp(-(z - torch.where(k, zmin[at], z)) / tau), torch.zeros_like(al))
                    acc.index_add_(0, at, torch.cat([w[:, None] * color_i, w[:, None]], 1))
                    lg.index_add_(0, at, torch.where(k, (1.0 - al).clamp(min=1e-6).log(), torch.zeros_like(al)))
    cover = (1.0 - lg.exp())[:, None]
    rgb = torch.where(acc[:, 3:] > 1e-8, acc[:, :3] / acc[:, 3:].clamp(min=1e-8), torch.ones_like(acc[:, :3]))
    img = (rgb * cover + (1.0 - cover)).clamp(0.0, 1.0).reshape(H, W, 3)
    return {"pos": pos, "cov": cov, "color": color, "image": img}
