"""The work that users of spacetime_gb300 have it do, as cases that can be timed.

Each case is one call (or one short sequence of calls) of the package's public
API, on inputs made from a seed: the camera's azimuth, the sky, the gas and the
first label index come from it, the sizes and rules from the case.

    still      render_draft: one frame by the kernel's rules, in any precision,
               with gas, a thin disc or neither, with one or several passes, and
               with the learned surrogate
    render     render: the CPU renderer's call (FP64, Schwarzschild)
    track      render_frames: a camera track in one call
    dolly      the layered engine on a camera that changes its radius from frame
               to frame, so each frame needs deflection fans of its own
    labels     Surrogate.generate: FP64 training labels
    train      Surrogate.train: AdamW steps on labels made before
    fluid      DiscFluidSim.step and .state: the live fluid disc

`exact` gives the 64-bit result of the cases that plain torch can follow in
some seconds: frames of one pass and at most EXACT_RAYS rays, labels, training
and the fluid.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from spacetime_gb300 import _abi, api, scene, surrogate
from spacetime_gb300.ship import free_fall_track

FOV = scene.lens_fov(24.0)
SKY = (1024, 512)
EXACT_RAYS = 70_000
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------

def listed():
    gas = dict(kind="still", scene="gas", a=0.9, r=15.0, incl=80.0, samples=1, landing=1, sigma=0.0,
               nr=256, nphi=64, nz=32)
    thin = dict(kind="still", scene="disc", a=0.9, r=15.0, incl=80.0, samples=1, landing=1, sigma=0.0)
    return [
        # a thumbnail of the Kerr + gas scene, as an editor redraws it while a slider moves
        dict(gas, name="thumbnail-gas-fp32-64x36", width=64, height=36, precision="fp32"),
        # render() as its reference is called: a small Schwarzschild frame with the thin disc
        dict(name="render-disc-fp64-320x180", kind="render", width=320, height=180, samples=1),
        # a reference-quality still to judge the fast precisions by
        dict(gas, name="still-gas-fp64-320x180", width=320, height=180, precision="fp64"),
        # the frame of the benchmark: Kerr, volumetric gas, full HD, single precision
        dict(gas, name="still-gas-fp32-1920x1080", width=1920, height=1080, precision="fp32"),
        # render_draft with its default four jittered passes, on a frame of odd sides
        dict(thin, name="draft-disc-fp32-4pass-961x541", width=961, height=541, precision="fp32", samples=2,
             landing=0),
        # a still with the FP64 guard steps near the photon ring
        dict(gas, name="still-gas-fp32g-960x540", width=960, height=540, precision="fp32g"),
        # a fall toward the hole, by render_frames' own defaults
        dict(name="track-disc-fp32g-16x640x360", kind="track", width=640, height=360, frames=16, r0=30.0, r1=4.0,
             precision="fp32g"),
        # a live view that moves in: layered engine, half-size layer, full-size photon ring
        dict(name="dolly-disc-fp32-2x1280x720", kind="dolly", width=1280, height=720, frames=2, half=True,
             ring=6.0, r=30.0),
        # the empty hole, with the trained network serving the pixels it is sure of
        dict(thin, name="still-surrogate-1920x1080", scene="empty", width=1920, height=1080, precision="fp32",
             sigma=4e-4),
        # training labels of the surrogate
        dict(name="labels-131072", kind="labels", n=131072, dt=0.02),
        # the surrogate's training loop at its recipe's batch
        dict(name="train-20x16384", kind="train", steps=20, batch=16384, rows=131072),
        # the fluid disc between two redraws, then its state for a plot
        dict(name="fluid-256x64x32-100", kind="fluid", nr=256, nphi=64, nz=32, steps=100, jacobi=8, dt=0.08),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def frame(lo, hi):
        w = log_int(lo, hi)
        return dict(width=w, height=max(9, min(w * 9 // 16, int(round(w * 9 / 16 * rng.uniform(0.8, 1.0))))))

    def grid():
        return dict(nr=rng.randint(64, 256), nphi=rng.randint(32, 64), nz=rng.randint(16, 32))

    kind = rng.choice(["still", "still", "fp64", "guarded", "passes", "render", "track", "dolly", "surrogate",
                       "labels", "train", "fluid"])
    a = round(rng.uniform(0.3, 0.99), 3)
    pose = dict(a=a, r=round(rng.uniform(12.0, 18.0), 2), incl=round(rng.uniform(60.0, 88.0), 1))
    one = dict(kind="still", samples=1, landing=1, sigma=0.0)
    if kind == "still":
        return dict(one, scene="gas", precision="fp32", **pose, **frame(48, 1800), **grid())
    if kind == "fp64":
        return dict(one, scene="gas", precision="fp64", **pose, **frame(32, 300), **grid())
    if kind == "guarded":
        return dict(one, scene="gas", precision=rng.choice(["fp32g", "fp32g_df"]), **pose, **frame(64, 900), **grid())
    if kind == "passes":
        pose["a"] = rng.choice([0.0, a])
        return dict(one, scene=rng.choice(["disc", "empty"]), precision="fp32", **pose, **frame(64, 960),
                    ) | dict(samples=2, landing=0)
    if kind == "render":
        return dict(kind="render", samples=1, **frame(32, 320))
    if kind == "track":
        return dict(kind="track", frames=rng.randint(2, 16), r0=30.0, r1=4.0, precision="fp32g", **frame(64, 640))
    if kind == "dolly":
        return dict(kind="dolly", frames=2, half=rng.random() < 0.5, ring=rng.choice([0.0, 6.0]),
                    r=round(rng.uniform(22.0, 34.0), 2), **frame(128, 1100))
    if kind == "surrogate":
        pose["a"] = round(rng.uniform(0.1, 0.98), 3)
        return dict(one, scene=rng.choice(["disc", "empty"]), precision="fp32", **pose, **frame(256, 1600),
                    ) | dict(sigma=rng.choice([2e-4, 4e-4]))
    if kind == "labels":
        return dict(kind="labels", n=log_int(1000, 131072), dt=0.02)
    if kind == "train":
        batch = 128 * log_int(1, 128)
        return dict(kind="train", steps=rng.randint(5, 20), batch=batch, rows=max(batch, log_int(8192, 131072)))
    return dict(kind="fluid", steps=log_int(10, 100), jacobi=rng.choice([2, 7, 8, 16, 24]), dt=0.08, **grid())


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------

_volumes: dict = {}


def _volume(nr, nphi, nz, inner, seed):
    """The gas of the benchmark scene, turned in azimuth by the seed."""
    key = (nr, nphi, nz, inner)
    if key not in _volumes:
        _volumes[key] = scene.make_volume(inner=inner, outer=25.0, nr=nr, nphi=nphi, nz=nz, scale_height=0.05)
    v = _volumes[key]
    turn = int(np.random.default_rng(seed).integers(1, nphi))
    return scene.Volume(np.roll(v.density, turn, axis=1), v.log_s_in, v.log_s_out, v.z_max, v.scale_height,
                        v.emission_scale, v.opacity_scale, v.march_stride)


def _camera(r, incl, a, seed):
    p = scene.kerr_position(r, incl, a)
    phi = np.random.default_rng(seed + 1).uniform(0.0, 2.0 * math.pi)
    c, s = math.cos(phi), math.sin(phi)
    return scene.Camera.look_at((c * p[0] - s * p[1], s * p[0] + c * p[1], p[2]), (0, 0, 0), (0, 0, 1), FOV)


def _sky(seed):
    return scene.make_sky(*SKY, n_stars=5000, seed=seed)


def _isco(a):
    z1 = 1 + (1 - a * a) ** (1 / 3) * ((1 + a) ** (1 / 3) + (1 - a) ** (1 / 3))
    z2 = math.sqrt(3 * a * a + z1 * z1)
    return 3 + z2 - math.sqrt((3 - z1) * (3 + z1 + 2 * z2))


def _still_scene(case, seed):
    """(hole, camera, disc, volume) of a still."""
    a = case["a"]
    bh = api.Kerr(1.0, a) if a else api.Schwarzschild(1.0)
    cam = _camera(case["r"], case["incl"], a, seed)
    inner = round(_isco(a), 2)
    disc = None if case["scene"] == "empty" else api.AccretionDisc(inner, 25.0)
    vol = _volume(case["nr"], case["nphi"], case["nz"], inner, seed) if case["scene"] == "gas" else None
    return bh, cam, disc, vol


def _render_camera(seed):
    """The camera of the CPU renderer's frame: 30 M out, 3 M above the disc."""
    phi = np.random.default_rng(seed + 1).uniform(0.0, 2.0 * math.pi)
    return scene.Camera.look_at((30.0 * math.sin(phi), -30.0 * math.cos(phi), 3.0), (0, 0, 0), (0, 0, 1), FOV)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "still":
        s["bh"], s["cam"], disc, vol = _still_scene(case, seed)
        s["ctx"] = api.Context(_sky(seed), disc=disc, volume=vol)
        s["extra"] = {}
        if case["sigma"] > 0:
            s["net"] = surrogate.load_trained()
            s["ctx"].set_surrogate(s["net"])
            s["extra"] = dict(surrogate=1, surrogate_sigma=case["sigma"])
    elif kind == "render":
        s["sky"], s["cam"] = _sky(seed), _render_camera(seed)
        s["ctx"] = api.Context(s["sky"], disc=api.AccretionDisc(), emitter=_abi.ST_EMIT_KEPLER)
    elif kind == "track":
        incl = 85.0 + np.random.default_rng(seed + 1).uniform(-1.0, 1.0)
        s["cams"] = free_fall_track(case["r0"], case["r1"], case["frames"], M=1.0, incl_deg=incl, fov=FOV)
        s["ctx"] = api.Context(_sky(seed), disc=api.AccretionDisc())
    elif kind == "dolly":
        s["ctx"] = api.Context(_sky(seed), disc=api.AccretionDisc())
        s["cams"] = [_camera(case["r"] * (1.0 - 0.02 * k), 84.3, 0.0, seed) for k in range(case["frames"])]
        w, h = case["width"], case["height"]
        s["p"] = s["ctx"].params(_abi.ST_SEM_DRAFT, width=w, height=h, samples=1, pixel_jitter=0, exit_landing=1,
                                 precision=_abi.ST_PREC_FP32)
        s["layer"] = ((w + 1) // 2, (h + 1) // 2) if case["half"] else None
    elif kind == "labels":
        s["net"] = surrogate.Surrogate(seed=seed % 1000)
        s["offset"] = _label_offset(seed)
    elif kind == "train":
        s["net"] = surrogate.Surrogate(seed=seed % 1000)
        s["net"].generate(case["rows"], offset=_label_offset(seed), copy=False)
    else:
        vol = _volume(case["nr"], case["nphi"], case["nz"], 2.32, seed)
        s["ctx"] = api.Context(_sky(seed), disc=api.AccretionDisc(2.32, 25.0), volume=vol)
        s["sim"] = api.DiscFluidSim(s["ctx"], vol, api.AccretionDisc(2.32, 25.0))
    return s


def _label_offset(seed):
    return (seed % 4096) * 131072


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "still":
        return api.render_draft(s["ctx"], s["cam"], s["bh"], width=s["width"], height=s["height"],
                                samples=s["samples"], precision=s["precision"], pixel_jitter=s["samples"] > 1,
                                exit_landing=s["landing"], **s["extra"])
    if kind == "render":
        return api.render(s["cam"], api.Schwarzschild(1.0), s["sky"], width=s["width"], height=s["height"],
                          samples=s["samples"], context=s["ctx"])
    if kind == "track":
        return api.render_frames(s["ctx"], s["cams"], api.Schwarzschild(1.0), width=s["width"], height=s["height"],
                                 precision=s["precision"], nmax=20000, exit_landing=1)
    if kind == "dolly":
        return [s["ctx"].render_layered_raw(c, api.Schwarzschild(1.0), s["p"], layer_size=s["layer"],
                                            ring_rmin=s["ring"]).image for c in s["cams"]]
    if kind == "labels":
        return s["net"].generate(s["n"], offset=s["offset"], dt=s["dt"])
    if kind == "train":
        hist = s["net"].train(s["steps"], batch=s["batch"], lr=1e-3, weight_decay=1e-6)
        return {"loss": hist, "params": s["net"].get_params()}
    s["sim"].step(dt=s["dt"], jacobi=s["jacobi"], nsteps=s["steps"])
    return s["sim"].state(volume=True)


# Flops of an RK4 step by the plain formulas, and steps and gas samples a ray
# takes on average in these scenes (counted by the kernels).
STEP_KERR, STEP_SCHW, GAS_SAMPLE = 578, 210, 100
STEPS_GAS, SAMPLES_GAS, STEPS_DRAFT, STEPS_RENDER, STEPS_TRACK, STEPS_LAYER = 1170, 516, 600, 1400, 700, 200


def work(case):
    kind = case["kind"]
    sky = SKY[0] * SKY[1] * 12
    if kind == "fluid":
        n = case["nr"] * case["nphi"]
        return {"bytes": case["steps"] * 4 * (19 * n + n * case["nz"]) + 4 * (3 * n + n * case["nz"]),
                "flops": case["steps"] * n * (500 + 8 * case["jacobi"] + case["nz"])}
    if kind == "labels":
        return {"bytes": case["n"] * 4 * (6 + 8 + 15), "flops": case["n"] * 1100 * STEP_KERR}
    if kind == "train":
        p = 200_710
        return {"bytes": case["steps"] * 4 * (case["batch"] * 14 + 6 * p),
                "flops": case["steps"] * (case["batch"] * 6 * p + 12 * p)}
    rays = case["width"] * case["height"] * case.get("frames", 1)
    out = 12 * rays
    rays *= case.get("samples", 1) ** 2
    if kind == "render":
        return {"bytes": sky + out, "flops": rays * STEPS_RENDER * STEP_SCHW}
    if kind == "track":
        return {"bytes": sky + out, "flops": rays * STEPS_TRACK * STEP_SCHW}
    if kind == "dolly":
        return {"bytes": sky + out, "flops": (rays // 4 if case["half"] else rays) * STEPS_LAYER * STEP_SCHW}
    step = STEP_KERR if case["a"] else STEP_SCHW
    if case["scene"] == "gas":
        vol = 4 * case["nr"] * case["nphi"] * case["nz"]
        return {"bytes": sky + vol + out, "flops": rays * (STEPS_GAS * step + SAMPLES_GAS * GAS_SAMPLE)}
    if case["sigma"] > 0:
        return {"bytes": sky + out, "flops": rays * (STEPS_DRAFT * step // 2 + 2 * 200_710)}
    return {"bytes": sky + out, "flops": rays * STEPS_DRAFT * step}


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch and numpy.
# ---------------------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "fluid":
        return _fluid64(case, seed)
    if kind == "labels":
        return _labels64(case["n"], _label_offset(seed), case["dt"])
    if kind == "train":
        return _train64(case, seed)
    if kind in ("still", "render") and case["samples"] == 1 and case["width"] * case["height"] <= EXACT_RAYS:
        if kind == "render":
            return _frame64(case, seed)
        if case["sigma"] == 0:
            return _frame64(case, seed)
    return None


def _dev(x):
    return torch.as_tensor(np.asarray(x), dtype=torch.float64, device=DEVICE)


def _dot(u, v):
    return (u * v).sum(0)


def _ks(pos, a):
    """Kerr-Schild r, the null vector l (3, n) and f / M at positions (3, n)."""
    x, y, z = pos
    w = _dot(pos, pos) - a * a
    r2 = (0.5 * (w + torch.sqrt(w * w + 4 * (a * z) ** 2))).clamp_min(1e-12)
    r = torch.sqrt(r2)
    d = r2 + a * a
    ell = torch.stack([(r * x + a * y) / d, (r * y - a * x) / d, z / r])
    return r, ell, 2 * r2 * r / (r2 * r2 + (a * z) ** 2)


def _rhs(s, pt, a):
    """dx, dp (6, n) of H = (-pt^2 + p^2 - f (l.p - pt)^2) / 2 for M = 1."""
    x, y, z, px, py, pz = s
    r, l, f = _ks(s[:3], a)
    r2, a2, z2 = r * r, a * a, z * z
    sig, d = r2 * r2 + a2 * z2, r2 + a2
    lp = _dot(l, s[3:]) - pt
    grad = torch.stack([x * r2 * r, y * r2 * r, z * r * d]) / sig
    dfdr = 2 * r2 * (3 * a2 * z2 - r2 * r2) / (sig * sig)
    dfdz = -4 * r2 * r * a2 * z / (sig * sig)
    dldr = (px * (x - 2 * r * l[0]) + py * (y - 2 * r * l[1])) / d - z * pz / r2
    direct = torch.stack([(r * px - a * py) / d, (a * px + r * py) / d, pz / r])
    dp = (0.5 * lp * lp * dfdr + f * lp * dldr) * grad + f * lp * direct
    dp[2] += 0.5 * lp * lp * dfdz
    return torch.cat([s[3:] - f * lp * l, dp])


def _rk4(y, pt, a, h, k1):
    k2 = _rhs(y + 0.5 * h * k1, pt, a)
    k3 = _rhs(y + 0.5 * h * k2, pt, a)
    k4 = _rhs(y + h * k3, pt, a)
    return y + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _land(yp, pt, a, h, target):
    """The state on the sphere |x| = target inside a step of size h from yp."""
    k1 = _rhs(yp, pt, a)
    lo, hi = torch.zeros_like(h), h.clone()
    rise = torch.linalg.vector_norm(_rk4(yp, pt, a, h, k1)[:3], dim=0) > target
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        beyond = (torch.linalg.vector_norm(_rk4(yp, pt, a, mid, k1)[:3], dim=0) > target) == rise
        lo, hi = torch.where(beyond, lo, mid), torch.where(beyond, mid, hi)
    return _rk4(yp, pt, a, 0.5 * (lo + hi), k1)


def _blackbody(T):
    lam = np.arange(380.0, 780.1, 5.0)
    lm = lam * 1e-9

    def bell(mu, s1, s2):
        return np.exp(-0.5 * ((lam - mu) / np.where(lam < mu, s1, s2)) ** 2)

    B = 1.0 / (lm ** 5 * (np.exp(0.014388 / (lm * T[:, None])) - 1.0))
    X = B @ (1.056 * bell(599.8, 37.9, 31.0) + 0.362 * bell(442.0, 16.0, 26.7) - 0.065 * bell(501.1, 20.4, 26.2))
    Y = B @ (0.821 * bell(568.8, 46.9, 40.5) + 0.286 * bell(530.9, 16.3, 31.1))
    Z = B @ (1.217 * bell(437.0, 11.8, 36.0) + 0.681 * bell(459.0, 26.0, 13.8))
    c = np.maximum(np.stack([3.2406 * X - 1.5372 * Y - 0.4986 * Z, -0.9689 * X + 1.8758 * Y + 0.0415 * Z,
                             0.0557 * X - 0.2040 * Y + 1.0570 * Z], 1), 0.0)
    return c / np.maximum(c.max(1, keepdims=True), 1e-10)


def _colour(T, table, half_up):
    x = (T.clamp(500.0, 30000.0) - 500.0) / 29500.0 * 1023
    return table[(torch.floor(x + 0.5) if half_up else torch.round(x)).long().clamp(0, 1023)].T


def _emitter(x, y, px, py, E, a, isco):
    """1 + z of the orbiting (inside the ISCO: plunging) emitter."""
    a2 = a * a
    isco = torch.as_tensor(isco, dtype=x.dtype, device=x.device)
    Ei = torch.sqrt(1 - 2 / (3 * isco))
    Li = 2 / (3 * math.sqrt(3)) * (1 + 2 * torch.sqrt(3 * isco - 2))
    s2 = x * x + y * y
    r = torch.sqrt((s2 - a2).clamp_min(1e-6))
    r32 = r * torch.sqrt(r)
    den = r32 - 3 * torch.sqrt(r) + 2 * a
    ut = (r32 + a) / (torch.sqrt(r32) * torch.sqrt(den.clamp_min(1e-2)))
    up = ut / (r32 + a)
    delta = r * r - 2 * r + a2
    inv = 1 / delta.clamp_min(1e-3)
    R = (Ei * (r * r + a2) - a * Li) ** 2 - delta * (r * r + (Li - a * Ei) ** 2)
    ur = -torch.sqrt(R.clamp_min(0)) / (r * r)
    utp = ((r * r + a2 + 2 * a2 / r) * Ei - 2 * a * Li / r) * inv + 2 * r * inv * ur
    upp = (2 * a * Ei / r + (1 - 2 / r) * Li) * inv + a * inv * ur
    orbit = r >= isco
    ur = torch.where(orbit, 0.0, ur)
    ut, up = torch.where(orbit, ut, utp), torch.where(orbit, up, upp)
    is2 = 1 / s2.clamp_min(1e-6)
    ux = ur * (r * x + a * y) * is2 - y * up
    uy = ur * (r * y - a * x) * is2 + x * up
    return (ut - (px * ux + py * uy) / torch.where(E.abs() > 1e-6, E, 1e-6)).clamp(0.1, 20)


def _planck(T):
    return 100 / (torch.exp(29622.4 / T.clamp_min(1.0)) - 1)


def _disc(s, pt, disc, a, isco, kepler, table):
    """(radiance (3, n), opacity) of the thin disc at crossing states s."""
    x, y = s[0], s[1]
    rad = torch.sqrt(x * x + y * y)
    R, Rin, Rout = rad / 2, disc[0] / 2, disc[1] / 2
    if kepler:
        f = 2 / rad
        c1 = f * (-pt + (x * s[3] + y * s[4]) / rad) / rad
        pc = torch.stack([s[3] - c1 * x, s[4] - c1 * y, s[5]])
        T = torch.exp(10.034259 - 0.375 * torch.log(R * R))
        v = (0.70710678 / torch.sqrt((R - 1).clamp_min(0.1))).clamp(0, 0.999)
        gam = 1 / torch.sqrt(1 - (v * v).clamp(0, 0.99))
        dop = gam * (1 + v * (-y * pc[0] + x * pc[1]) / rad / torch.sqrt(_dot(pc, pc)))
        obs = T / (dop / torch.sqrt((1 - 1 / R.clamp_min(1.0)).clamp_min(0.01))).clamp_min(0.1)
        plunge = 1.0
    else:
        T = torch.exp(10.034259 - 0.375 * torch.log((rad.clamp_min(isco) / 2) ** 2))
        plunge = torch.where(rad < isco, (rad / isco) ** 3, 1.0)
        obs = T / _emitter(x, y, s[3], s[4], -pt, a, isco)
    op = ((R * R - Rin * Rin) * 0.3).clamp(0, 1) * (T / 1000).clamp(0, 1) * plunge
    op = torch.where((rad > disc[0]) & (rad < disc[1]), op, 0.0)
    return _planck(obs) * _colour(obs, table, not kepler) * op, op


def _density(vol, meta, s, phi, z):
    nz, nphi, nr = vol.shape
    li, lo, zmax = meta
    ls = torch.log(s.clamp_min(1e-6))
    fr = (ls - li) / (lo - li) * (nr - 1)
    fp = torch.where(phi < 0, phi + 2 * math.pi, phi) / (2 * math.pi) * nphi
    fz = (z + zmax) / (2 * zmax) * (nz - 1)
    i = torch.floor(fr).long().clamp(0, nr - 2)
    j = torch.floor(fp).long()
    k = torch.floor(fz).long().clamp(0, nz - 2)
    tr, tp, tz = fr - i, fp - j, fz - k
    j, j1 = j % nphi, (j + 1) % nphi

    def row(jj, kk):
        return vol[kk, jj, i] * (1 - tr) + vol[kk, jj, i + 1] * tr

    lower = row(j, k) * (1 - tp) + row(j1, k) * tp
    upper = row(j, k + 1) * (1 - tp) + row(j1, k + 1) * tp
    return torch.where((ls > li) & (ls < lo) & (z.abs() < zmax), lower * (1 - tz) + upper * tz, 0.0)


def _gas(yp, y, r2, seg, st, gas, a, isco, table, dt):
    """The gas along one step; st: rows march, alpha, r, g, b."""
    vol, meta, emis, opac, stride, rb2 = gas
    ds = stride * dt
    go = (st[1] > 0.003) & (torch.minimum(r2, _dot(y[:3], y[:3])) < rb2) & (seg < 64)
    t = ds - st[0]
    none = go & (t > seg)
    st[0] = torch.where(none, st[0] + seg, st[0])
    march = go & ~none
    live = march.clone()
    while bool(live.any()):
        fs = t / seg
        q = yp + fs * (y - yp)
        s = torch.sqrt(q[0] ** 2 + q[1] ** 2)
        rho = _density(vol, meta, s, torch.atan2(q[1], q[0]), q[2])
        lit = live & (rho > 1e-4) & (s > 1e-6)
        T = torch.exp(10.034259 - 0.375 * torch.log(((s.clamp_min(isco) / 2) ** 2).clamp_min(1e-6)))
        rho = torch.where(s < isco, rho * (s / isco) ** 3, rho)
        obs = T / _emitter(q[0], q[1], q[3], q[4], st[5], a, isco)
        aa = torch.where(lit, 1 - torch.exp(-opac * rho * ds), 0.0)
        st[2:5] += torch.where(lit, st[1] * aa * _planck(obs) * emis * _colour(obs, table, True), 0.0)
        st[1] *= 1 - aa
        t = torch.where(live, t + ds, t)
        live = live & (t <= seg) & (st[1] > 0.003)
    st[0] = torch.where(march, seg - (t - ds), st[0])
    return march & (st[1] < 0.003)


def _captured(s, pt, a):
    """Bardeen's launch test: an ingoing ray without a turning point outside the horizon."""
    r, _, _ = _ks(s[:3], a)
    E, ct = -pt, s[2] / r
    s2 = (1 - ct * ct).clamp_min(1e-8)
    L = s[0] * s[4] - s[1] * s[3]
    pth = ct / torch.sqrt(s2) * (s[0] * s[3] + s[1] * s[4]) - r * torch.sqrt(s2) * s[5]
    lam, eta = L / E, (pth * pth + ct * ct * (L * L / s2 - a * a * E * E)) / (E * E)
    v = _rhs(s, pt, a)
    ingoing = r * r * (s[0] * v[0] + s[1] * v[1]) + (r * r + a * a) * s[2] * v[2] < 0
    c2, c1, c0 = a * a - lam * lam - eta, 2 * (eta + (lam - a) ** 2), -a * a * eta
    p, q = 0.5 * c2, 0.25 * c1
    D = 0.25 * q * q + p ** 3 / 27
    sq = torch.sqrt(D.clamp_min(0))
    u1, u2 = -0.5 * q + sq, -0.5 * q - sq
    one = torch.sign(u1) * u1.abs().clamp_min(1e-30) ** (1 / 3) + torch.sign(u2) * u2.abs().clamp_min(1e-30) ** (1 / 3)
    m = 2 * torch.sqrt((-p / 3).clamp_min(1e-300))
    t = torch.acos((3 * q / (p * m)).clamp(-1, 1)) / 3
    turn, graze = torch.zeros_like(D, dtype=torch.bool), torch.zeros_like(D, dtype=torch.bool)
    rp = 1 + torch.sqrt((1 - a * a + 0 * D).clamp_min(0))
    for k in range(3):
        rc = torch.where(D >= 0, one, m * torch.cos(t - 2.0943951023931953 * k))
        inside = (rc > rp) & (rc < r)
        Rv = ((rc * rc + c2) * rc + c1) * rc + c0
        turn |= inside & (Rv <= 0)
        graze |= inside & (Rv.abs() < 0.08 * (rc ** 4).clamp_min(1.0))
    return ingoing & ~turn, ingoing & graze


def _photon_orbit(a):
    return 2.0 * (1.0 + np.cos((2.0 / 3.0) * np.arccos(-a)))


def _trace(y, pt, a, draft, kerr, dt, r_esc, nmax, tspan, landing, disc=None, gas=None, isco=6.0, table=None,
           cross=False):
    """Integrates rays (6, n); returns end states, flags and light by ray.

    `a` is a number or one value a ray; r_esc a number or one value a ray."""
    n = y.shape[1]
    dev = y.device
    a = torch.as_tensor(a, dtype=torch.float64, device=dev).expand(n)
    r_esc = torch.as_tensor(r_esc, dtype=torch.float64, device=dev).expand(n)
    nmax = torch.as_tensor(nmax, dtype=torch.float64, device=dev).expand(n)
    rk = (0.995 * _dev(_photon_orbit(a.cpu().numpy()))).float()
    rkill2 = (rk * rk).double()
    one = not bool((a != a[0]).any())
    full = dict(y=y.clone(), esc=torch.zeros(n, dtype=torch.bool, device=dev),
                cap=torch.zeros(n, dtype=torch.bool, device=dev), light=torch.zeros(6, n, dtype=torch.float64, device=dev),
                steps=torch.zeros(n, dtype=torch.float64, device=dev),
                cross=torch.full((5, n), -1.0, dtype=torch.float64, device=dev))
    full["light"][1] = 1.0
    full["light"][5] = -pt
    idx = torch.arange(n, device=dev)
    lands = []
    r0 = torch.linalg.vector_norm(y[:3], dim=0)
    floor = torch.where(r0 > 2.05, 2.0, 0.3)
    prev, lam, st = torch.full_like(r0, -1.0), torch.zeros_like(r0), full["light"].clone()
    crossed = full["cross"].clone()
    alive = torch.ones(n, dtype=torch.bool, device=dev)
    A = float(a[0]) if one else a
    step = 0
    while idx.numel():
        r2 = _dot(y[:3], y[:3])
        r = torch.sqrt(r2)
        end = alive & (step >= nmax)
        done = end.clone()
        if draft and kerr:
            ks2 = _ks(y[:3], A)[0] ** 2
            kill = alive & ~done & (ks2 < rkill2)
        elif draft:
            near = r < 3.2
            kill = alive & ~done & near & ((r < floor) | ((r < 2.95) & (prev > 0) & (r < prev - 1e-4)))
            prev = torch.where(alive & near, r, prev)
        out = alive & ~done & ((r > r_esc) if draft else (r >= r_esc))
        if draft:
            out &= ~kill
        else:
            end = alive & ~out & (lam >= tspan)
            kill = alive & ~out & ~end & (r < 2.95) & (prev > 0) & (r < prev - 1e-4)
            prev = torch.where(alive, r, prev)
            done |= end
        full["esc"][idx[out]] = True
        full["cap"][idx[kill]] = True
        alive = alive & ~(done | kill | out)
        cap = torch.where(r2 < gas[5], 2.0, 8.0) if gas else 8.0
        h = dt * torch.minimum((0.16 * r).clamp_min(1.0), torch.as_tensor(cap, dtype=r.dtype, device=dev))
        if draft and kerr:
            h = h * (0.12 + 0.88 * ((ks2 - rkill2) / rkill2.clamp_min(1e-6)).clamp(0, 1))
        if not draft:
            h = torch.minimum(h, tspan - lam)
        h = torch.where(alive, h, 0.0)
        k1 = _rhs(y, pt, A)
        yn = torch.where(alive, _rk4(y, pt, A, h, k1), y)
        bad = alive & ~torch.isfinite(yn).all(0)
        full["cap"][idx[bad]] = True
        full["steps"][idx] += alive
        alive = alive & ~bad
        if gas:
            seg = torch.where(alive, h * torch.linalg.vector_norm(k1[:3], dim=0).clamp_min(1e-20), 1e9)
            alive = alive & ~_gas(y, yn, r2, seg, st, gas, A, isco, table, dt)
        elif disc or cross:
            hit = alive & (y[2] * yn[2] < 0) & ((st[1] > 0.001) | (not draft))
            if bool(hit.any()):
                w = hit.nonzero()[:, 0]
                fr = y[2][w] / (y[2][w] - yn[2][w])
                s = y[:, w] + fr * (yn[:, w] - y[:, w])
                if disc:
                    c, op = _disc(s, pt[w], disc, A if one else A[w], isco, not draft, table)
                    st[2:5, w] += c * st[1][w]
                    st[1, w] *= 1 - op
                if cross:
                    first = crossed[0][w] < 0
                    crossed[:, w[first]] = torch.stack([torch.sqrt(s[0] ** 2 + s[1] ** 2), s[0], s[1], s[3], s[4]])[:, first]
        rn = torch.linalg.vector_norm(yn[:3], dim=0)
        if draft:
            bound = alive & (rn > r_esc) if landing else torch.zeros_like(alive)
            target = r_esc
        else:
            inner = alive & (rn <= 2.00001)
            bound = inner | (alive & (rn >= r_esc))
            target = torch.where(inner, 2.00001, r_esc)
            full["cap"][idx[inner]] = True
            lam = lam + h
        if bool(bound.any()):
            w = bound.nonzero()[:, 0]
            lands.append((idx[w], y[:, w], pt[w], a[w], h[w], target[w]))
            full["esc"][idx[w]] = True
        alive = alive & ~bound
        y = yn
        step += 1
        if step % 32 == 0 or not bool(alive.any()):
            # write back what has ended, keep the rest
            full["y"][:, idx] = y
            full["light"][:, idx] = st
            full["cross"][:, idx] = crossed
            k = alive.nonzero()[:, 0]
            y, pt, idx, prev, lam, st, crossed = y[:, k], pt[k], idx[k], prev[k], lam[k], st[:, k], crossed[:, k]
            a, r_esc, nmax, rkill2, floor, alive = a[k], r_esc[k], nmax[k], rkill2[k], floor[k], alive[k]
            A = A if one else a
    if lands:
        i = torch.cat([x[0] for x in lands])
        full["y"][:, i] = _land(torch.cat([x[1] for x in lands], 1), *(torch.cat([x[m] for x in lands]) for m in (2, 3, 4, 5)))
    full["esc"] &= ~full["cap"]
    return full


def _tetrad(cam, a):
    """Rows u, forward, right, up of an observer at rest (static, or the ZAMO blend near the hole)."""
    pos = torch.as_tensor(cam.pos, dtype=torch.float64)
    r, l, f = (v.numpy() for v in _ks(pos[:, None], a))
    r, l, f = float(r[0]), l[:, 0], float(f[0])

    def g(u, v):
        return -u[0] * v[0] + u[1:] @ v[1:] + f * (u[0] + l @ u[1:]) * (v[0] + l @ v[1:])

    if a == 0.0:
        E = math.sqrt(max(0.2, 1 - f))
        v = -math.sqrt(max(E * E - (1 - f), 0.0))
        w = (1 - E * (E - v)) / (E - v)
        u = np.concatenate([[E + f * (E + w)], (w - f * (E + w)) * l])
    else:
        assert f <= 0.72
        u = np.array([1 / math.sqrt(1 - f), 0, 0, 0])
    rows = [u]
    for e in (cam.fwd, cam.right, cam.up_local):
        v = np.concatenate([[0.0], e])
        v = v + g(v, u) * u
        for k in rows[1:]:
            v = v - g(v, k) * k
        rows.append(v / math.sqrt(g(v, v)))
    return rows


def _lower(x, q, a):
    """Covariant momentum (state (6, n), p_t) of tangents q (4, n) at x (3, n)."""
    _, l, f = _ks(x, a)
    lq = q[0] + _dot(l, q[1:])
    return torch.cat([x, q[1:] + f * lq * l]), -q[0] + f * lq


def _nmax(r_esc, dt):
    n = np.ceil((75.0 + 6.5 * np.log(np.float32(r_esc))) / float(np.float32(dt)))
    return np.clip(n, 1000, 40000)


def _frame64(case, seed):
    draft = case["kind"] == "still"
    if draft:
        bh, cam, disc, vol = _still_scene(case, seed)
        a = bh.a
    else:
        cam, disc, vol, a = _render_camera(seed), api.AccretionDisc(), None, 0.0
    w, h, dt = case["width"], case["height"], 0.02
    u, Ef, Er, Eu = (_dev(v)[:, None] for v in _tetrad(cam, a))
    shift = 0.0 if draft else 0.5
    i = (_dev(np.arange(w)) + 0.5 + shift - w / 2) / (h / 2) * FOV
    j = (_dev(np.arange(h)) + 0.5 + shift - h / 2) / (h / 2) * FOV
    dy, dx = torch.meshgrid(j, i, indexing="ij")
    dx, dy = dx.reshape(-1), dy.reshape(-1)
    nu = torch.sqrt(dx * dx + dy * dy + 1)
    q = (Ef + dx * Er + dy * Eu) / nu - u
    y, pt = _lower(_dev(cam.pos)[:, None].expand(3, w * h).contiguous(), q, a)
    rpos = float(np.linalg.norm(cam.pos))
    table = _blackbody(np.linspace(500.0, 30000.0, 1024)) / _blackbody(np.array([6500.0]))
    table = _dev(table.astype(np.float32))
    gas = None
    if vol is not None:
        gas = (_dev(vol.density), (vol.log_s_in, vol.log_s_out, vol.z_max), float(np.float32(vol.emission_scale)),
               float(np.float32(vol.opacity_scale)), vol.march_stride, math.exp(vol.log_s_out) ** 2 + vol.z_max ** 2)
    r_esc = float(np.float32(2 * max(rpos, 15.0))) if draft else max(5 * rpos, 100.0)
    t = _trace(y, pt, a, draft, a != 0.0, dt, r_esc, float(_nmax(r_esc, dt)) if draft else 50000,
               max(10 * rpos, 500.0), case.get("landing", 1), None if disc is None else (disc.inner_radius, disc.outer_radius),
               gas, _isco(a), table)
    rf = torch.linalg.vector_norm(t["y"][:3], dim=0)
    black = t["cap"] | (rf < (4.0 if draft else 2.1))
    if draft and a:
        black |= _captured(y, pt, a)[0]
    v = _rhs(t["y"], pt, a)[:3]
    d = v / torch.linalg.vector_norm(v, dim=0)
    sky = _dev(_sky(seed))
    H, W = sky.shape[:2]
    xf = torch.atan2(d[1], d[0])
    xf = torch.where(xf < 0, xf + 2 * math.pi, xf) / (2 * math.pi) * (W - 1)
    yf = torch.acos(d[2].clamp(-1, 1)) / math.pi * (H - 1)
    x0, y0 = torch.floor(xf).long().clamp(0, W - 1), torch.floor(yf).long().clamp(0, H - 1)
    x1, y1 = (x0 + 1).clamp(max=W - 1), (y0 + 1).clamp(max=H - 1)
    fx, fy = (xf - x0)[:, None], (yf - y0)[:, None]
    s = (sky[y0, x0] * (1 - fx) + sky[y0, x1] * fx) * (1 - fy) + (sky[y1, x0] * (1 - fx) + sky[y1, x1] * fx) * fy
    rgb = t["light"][2:5].T + torch.where(black[:, None], 0.0, t["light"][1][:, None] * s)
    return rgb.reshape(h, w, 3).cpu()


def _sobol(idx):
    """Five dimensions of the Sobol sequence at integer indices, 24 bits each."""
    out = []
    for s, poly, m0 in ((0, 0, []), (1, 0, [1]), (2, 1, [1, 3]), (3, 1, [1, 3, 1]), (3, 2, [1, 1, 1])):
        m = list(m0) if s else [1] * 32
        for k in range(len(m), 32):
            v = m[k - s] ^ (m[k - s] << s)
            for j in range(1, s):
                if (poly >> (s - 1 - j)) & 1:
                    v ^= m[k - j] << j
            m.append(v)
        x = np.zeros(idx.shape, np.uint32)
        for k in range(32):
            x ^= np.where((idx >> np.uint32(k)) & np.uint32(1), np.uint32((m[k] << (31 - k)) & 0xFFFFFFFF), np.uint32(0))
        out.append(((x >> np.uint32(8)).astype(np.float32) + np.float32(0.5)) * np.float32(1 / 16777216))
    return out


def _labels64(n, offset, dt):
    u0, u1, u2, u3, u4 = _sobol((np.arange(n, dtype=np.int64) + offset + 1).astype(np.uint32))
    r, th, a = 4 + 46 * u0.astype(float), math.pi / 2 * u1.astype(float), 0.99 * u2.astype(float)
    c = 0.25881904510252074
    near, far = (u3 / np.float32(0.8)).astype(float), ((u3 - np.float32(0.8)) / np.float32(0.2)).astype(float)
    ca = np.where(u3 < np.float32(0.8), 1 - near * (1 - c), c - far * (1 + c))
    sa = np.sqrt(np.maximum(1 - ca * ca, 0))
    ph = 6.283185307179586 * u4.astype(float)
    nv = np.stack([-ca, sa * np.cos(ph), sa * np.sin(ph)])
    pos = np.stack([np.sqrt(r * r + a * a) * np.sin(th), 0 * r, r * np.cos(th)])
    rpos = np.linalg.norm(pos, axis=0)
    ct = pos[2] / rpos
    sn = np.sqrt(np.maximum(1 - ct * ct, 0))
    axes = [np.stack([pos[0] / rpos, 0 * r, ct]), np.stack([ct, 0 * r, -sn]), np.stack([0 * r, 1 + 0 * r, 0 * r])]
    x, A = _dev(pos), _dev(a)
    _, l, f = _ks(x, A)

    def g(p, q):
        return -p[0] * q[0] + _dot(p[1:], q[1:]) + f * (p[0] + _dot(l, p[1:])) * (q[0] + _dot(l, q[1:]))

    u = torch.cat([(1 / torch.sqrt(1 - f))[None], torch.zeros_like(x)])
    E = []
    for e in axes:
        v = torch.cat([torch.zeros_like(f)[None], _dev(e)])
        v = v + g(v, u) * u
        for k in E:
            v = v - g(v, k) * k
        E.append(v / torch.sqrt(g(v, v)))
    q = _dev(nv[0]) * E[0] + _dev(nv[1]) * E[1] + _dev(nv[2]) * E[2] - u
    y, pt = _lower(x, q, A)
    cap0, graze = _captured(y, pt, A)
    v0 = _rhs(y, pt, A)[:3]
    d0 = v0 / torch.linalg.vector_norm(v0, dim=0)
    r_esc = (2 * np.maximum(rpos, 15.0)).astype(np.float32).astype(float)
    nm = np.clip(np.ceil((75 + 6.5 * np.log(r_esc)) / dt), 1000, 40000)
    t = _trace(y, pt, A, True, True, dt, _dev(r_esc), _dev(nm), 0.0, True, cross=True)
    v = _rhs(t["y"], pt, A)[:3]
    d = v / torch.linalg.vector_norm(v, dim=0)
    isco = np.array([_isco(k) for k in a])
    rc = t["cross"][0]
    hit = rc > 0
    gc = torch.zeros_like(rc)
    k = hit.nonzero()[:, 0]
    if k.numel():
        gc[k] = 1 / _emitter(*t["cross"][1:, k], -pt[k], A[k], _dev(isco)[k])
    budget = ~t["esc"] & ~t["cap"]
    ok = t["esc"] & ~cap0
    xh = x / _dev(rpos)
    cc = _dot(xh, d0)
    tt = d0 - cc * xh
    sn = torch.linalg.vector_norm(tt, dim=0)
    et = tt / sn
    en = torch.linalg.cross(xh, et, dim=0)
    D = torch.atan2(_dot(d, et), _dot(d, xh)) - torch.atan2(sn, cc)
    D = D - 2 * math.pi * torch.floor((D + math.pi / 2) / (2 * math.pi))
    tilt = torch.asin(_dot(d, en).clamp(-1, 1))
    X = torch.stack([(_dev(r) - 27) / 23, _dev(th) / 0.78539816 - 1, A / 0.495 - 1, *_dev(nv)], 1)
    zero = torch.zeros_like(D)
    T = torch.stack([torch.where(ok, D, zero), torch.where(ok, tilt, zero), zero,
                     torch.where(hit, (10 / rc).clamp(max=5.0), zero) - 1, torch.where(hit, gc - 1, zero), ok.double(),
                     hit.double(), zero], 1)
    bits = (_abi.ST_RAY_CAPTURED * t["cap"].double() + _abi.ST_RAY_ESCAPED * t["esc"].double()
            + _abi.ST_RAY_BUDGET * budget.double() + _abi.ST_RAY_BCAPT * cap0.double() + _abi.ST_RAY_GRAZE * graze.double())
    raw = torch.stack([_dev(r), _dev(th), A, *_dev(nv), bits, t["steps"], *d, rc, *d0], 1)
    return [X.cpu(), T.cpu(), raw.cpu()]


def _train64(case, seed):
    """AdamW on the same rows and from the same weights, every number in 64 bits."""
    s = prepare(case, seed)  # the inputs: initial weights and label rows
    X, T, _ = s["net"].generate(case["rows"], offset=_label_offset(seed))
    X, T = _dev(X), _dev(T)
    P = _dev(s["net"].get_params()).requires_grad_()
    shapes = [(256, 6), (256,), (256, 256), (256,), (256, 256), (256,), (256, 256), (256,), (6, 256), (6,)]
    sizes = [math.prod(k) for k in shapes]
    decay = torch.cat([torch.full((n,), float(len(k) == 2), dtype=torch.float64, device=DEVICE)
                       for n, k in zip(sizes, shapes)])
    m, v, hist = torch.zeros_like(P), torch.zeros_like(P), []
    lr, wd, B = 1e-3, 1e-6, case["batch"]
    nb = case["rows"] // B
    for k in range(case["steps"]):
        at = (k * 7919) % nb * B
        x, t = X[at:at + B], T[at:at + B]
        W = [p.view(q) for p, q in zip(P.split(sizes), shapes)]
        for L in range(0, 8, 2):
            x = torch.nn.functional.silu(x @ W[L].T + W[L + 1])
        o = x @ W[8].T + W[9]
        sg = o[:, 5].clamp(-30, 12)
        e2 = (o[:, 0] - t[:, 0]) ** 2 + (o[:, 1] - t[:, 1]) ** 2
        loss = (t[:, 5] * (0.5 * e2 * torch.exp(-sg) + sg) + (o[:, 3] - t[:, 3]) ** 2
                + t[:, 6] * (o[:, 4] - t[:, 4]) ** 2).mean()
        G, = torch.autograd.grad(loss, P)
        hist.append(float(loss))
        m = 0.9 * m + 0.1 * G
        v = 0.999 * v + 0.001 * G * G
        with torch.no_grad():
            P = P * (1 - lr * wd * decay)
            P = P - lr * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
        P.requires_grad_()
    return {"loss": np.array(hist), "params": P.detach().cpu()}


def _fluid64(case, seed):
    vol = _volume(case["nr"], case["nphi"], case["nz"], 2.32, seed)
    nr, nphi, nz = vol.shape
    dt, forcing, drag, relax = float(np.float32(case["dt"])), 6.0, float(np.float32(0.15)), float(np.float32(0.05))
    dens = _dev(vol.density[(nz + 1) // 2 - 1])
    dens = dens / dens.max()
    s = np.exp(vol.log_s_in + np.arange(nr) / (nr - 1) * (vol.log_s_out - vol.log_s_in))
    R, Rin = s / 2, 2.32 / 2
    base = np.clip((R * R - Rin * Rin) * 0.3, 0, 1) * np.clip(np.exp(10.034259 - 0.375 * np.log(R * R)) / 1000, 0, 1)
    z = -vol.z_max + np.arange(nz) / (nz - 1) * 2 * vol.z_max
    env = _dev(np.exp(-z[:, None] ** 2 / (2 * (vol.scale_height * s) ** 2)))
    shear = _dev(np.sqrt(1 / s ** 3) * nphi / (2 * math.pi))
    base = _dev(base).expand(nphi, nr)
    I = _dev(np.arange(1, nr + 1)).expand(nphi, nr)
    J = _dev(np.arange(1, nphi + 1))[:, None].expand(nphi, nr)

    def hash01(i, j, k):
        i, j, k = (v & 0xFFFFFFFF for v in (i, j, k))
        h = (i * 0x8DA6B343 & 0xFFFFFFFF) ^ (j * 0xD8163841 & 0xFFFFFFFF) ^ (k * 0xCB1AB31F & 0xFFFFFFFF)
        h = ((h ^ (h >> 13)) * 0x9E3779B9) & 0xFFFFFFFF
        return ((h ^ (h >> 16)) & 0xFFFFFF).double() * 5.9604645e-8

    def noise(x, y, t):
        x, y, t = torch.broadcast_tensors(x, y, torch.full_like(x, t))
        fx, fy, fz = torch.floor(x), torch.floor(y), torch.floor(t)
        ix, iy, iz = fx.long(), fy.long(), fz.long()
        fx, fy, fz = ((v * v * (3 - 2 * v)) for v in (x - fx, y - fy, t - fz))
        c = [[hash01(ix, iy + b, iz + e) * (1 - fx) + hash01(ix + 1, iy + b, iz + e) * fx for b in (0, 1)] for e in (0, 1)]
        lo, hi = (c[e][0] * (1 - fy) + c[e][1] * fy for e in (0, 1))
        return lo * (1 - fz) + hi * fz

    def corners(x, y):
        x = x.clamp(1, nr)
        i = torch.floor(x).long().clamp(1, nr - 1)
        yw = y - nphi * torch.floor((y - 1) / nphi)
        j = torch.floor(yw)
        return i - 1, (j.long() - 1) % nphi, j.long() % nphi, x - i, yw - j

    def sample(f, q):
        i, j0, j1, tx, ty = q
        lo = f[j0, i] * (1 - tx) + f[j0, i + 1] * tx
        hi = f[j1, i] * (1 - tx) + f[j1, i + 1] * tx
        return lo * (1 - ty) + hi * ty

    def up(f):
        return torch.cat([f[:, 1:], f[:, -1:]], 1)

    def down(f):
        return torch.cat([f[:, :1], f[:, :-1]], 1)

    vu, vv, t, e = torch.zeros_like(dens), torch.zeros_like(dens), 0.0, 0.35
    edge = (torch.minimum(I - 1, nr - I) * 0.125).clamp(0, 1)
    damp = math.exp(-drag * dt)
    for _ in range(case["steps"]):
        q = corners(I - dt * vu, J - dt * (vv + shear))
        px, py, pz = I * 0.085, J * 0.085, t * 0.35
        fu = (noise(px, py + e, pz) - noise(px, py - e, pz)) / (2 * e)
        fv = -(noise(px + e, py, pz) - noise(px - e, py, pz)) / (2 * e)
        u = (sample(vu, q) + dt * forcing * fu * edge) * damp * edge
        v = (sample(vv, q) + dt * forcing * fv * edge) * damp
        div = 0.5 * (up(u) - down(u) + v.roll(-1, 0) - v.roll(1, 0))
        p = torch.zeros_like(u)
        for _ in range(2 * ((case["jacobi"] + 1) // 2)):
            p = 0.25 * (up(p) + down(p) + p.roll(-1, 0) + p.roll(1, 0) - div)
        vu, vv = u - 0.5 * (up(p) - down(p)), v - 0.5 * (p.roll(-1, 0) - p.roll(1, 0))
        q = corners(I - dt * vu, J - dt * (vv + shear))
        d1 = sample(dens, q)
        i, j0, j1 = q[:3]
        four = torch.stack([dens[j0, i], dens[j0, i + 1], dens[j1, i], dens[j1, i + 1]])
        d2 = sample(d1, corners(I + dt * vu, J + dt * (vv + shear)))
        adv = torch.minimum(torch.maximum(d1 + 0.5 * (dens - d2), four.min(0).values), four.max(0).values)
        tgt = base * torch.exp(1.2 * (2 * noise(I * 0.11, J * 0.11, t * 0.25) - 1))
        dens = (adv + relax * dt * (tgt - adv)).clamp_min(0)
        t += dt
    return {"vu": vu.cpu(), "vv": vv.cpu(), "dens": dens.cpu(), "t": t, "volume": (env[:, None, :] * dens).cpu()}
