"""Workloads that time this framework through its public entry points.

Each case is one call (or the short fixed sequence of calls) that a user's
program makes: a frame of the image tracer at a precision and integrator, a
batch of uneven frames, a frame of the learned surrogate, a training step, a
radiative-transfer image, a frame of the render launch ABI, its
post-processing, and the batched geodesic API.

``prepare`` makes what such a program holds before the call (scenes, output
buffers, the sky, the medium, the network), ``run`` makes the call, ``exact``
gives the same outputs in 64 bits from formulas written out here, where an
output has a value that does not depend on the integrator's own steps.
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

from blackhole_b200 import kerr, legacy, rt
from blackhole_b200 import surrogate as S

WEIGHTS = Path(__file__).resolve().parent.parent / "blackhole_b200" / "data" / "surrogate_c4.npz"
INTEGRATORS = {"rk4": 0, "dp45": 1, "closed": 2}
# the outputs of a program that only shades the disk: no azimuths
DISK_FIELDS = ("cls", "n_cross", "r_hit", "g", "flux", "intensity")
ALL_FIELDS = ("cls", "steps", "n_cross", "r_hit", "phi_hit", "g", "flux", "intensity", "theta_inf", "phi_inf")
INT_FIELDS = ("cls", "steps", "n_cross")
SIDES = (64, 128, 256, 512)  # frame sides of the uneven batches
MLP_FLOPS = 2.0 * (134 * 256 + 3 * 256 * 256 + 256 * 16)  # one row of the network


def listed():
    return [
        # the smallest call: a thumbnail re-traced while a scene is being set up; launches and one ray's chain count
        dict(name="preview_64x48", kind="frame", integrator="dp45", precision="fp64", width=64, height=48,
             crossings=3, fields="all", sky=False, spin=0.9, incl=60.0),
        # a program on the batched geodesic API: some thousands of rays, first-order scheme with fixed steps
        dict(name="rays_4096", kind="rays", n=4096, steps=1500, spin=0.9),
        # the default scene of the library: fixed-step RK4, opaque disk
        dict(name="rk4_256", kind="frame", integrator="rk4", precision="fp64", width=256, height=256,
             crossings=1, fields="all", sky=False, spin=0.9, incl=60.0),
        # an ordinary FP64 frame at the bridge's preview size, transparent disk in front of a sky
        dict(name="dp45_640x360", kind="frame", integrator="dp45", precision="fp64", width=640, height=360,
             crossings=3, fields="all", sky=True, spin=0.5, incl=75.0),
        # many frames of uneven size in one persistent launch, mixed precision
        dict(name="batch_48", kind="batch", frames=48, crossings=3, sky=True),
        # an odd-sized frame in closed form, every output
        dict(name="closed_1279x721", kind="frame", integrator="closed", precision="fp64", width=1279, height=721,
             crossings=3, fields="all", sky=False, spin=0.94, incl=80.0),
        # the headline frame: 2048^2 through the learned surrogate, every output
        dict(name="surrogate_2048", kind="surrogate", width=2048, height=2048, crossings=1, fields="all", spin=0.9,
             incl=60.0),
        # forward and backward of one training batch
        dict(name="train_16384", kind="train", batch=16384),
        # the image of a volumetric emitter, both precisions
        dict(name="transfer_512", kind="transfer", precision="mixed", width=512, height=512, spin=0.94, incl=17.0),
        dict(name="transfer_fp64_160", kind="transfer", precision="fp64", width=160, height=160, spin=0.94,
             incl=17.0),
        # a full-HD frame of the render launch ABI, and the bloom and tone mapping of such a frame
        dict(name="render_1920x1080", kind="render", width=1920, height=1080, spin=0.9, incl=60.0, distance=10.0),
        dict(name="post_1920x1080", kind="post", width=1920, height=1080, bloom=0.5),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def shape(lo, hi):  # width and height of a frame of lo to hi pixels
        n, aspect = log_int(lo, hi), rng.uniform(0.5, 2.0)
        w = max(1, int(round(math.sqrt(n * aspect))))
        return w, max(1, n // w)

    spin, incl = round(rng.uniform(0.0, 0.998), 4), round(rng.uniform(5.0, 88.0), 3)
    kind = rng.choice(("frame", "frame", "closed", "rays", "batch", "surrogate", "train", "forward", "transfer",
                       "render", "post"))
    if kind == "rays":
        return dict(kind="rays", n=log_int(1, 60000), steps=log_int(100, 2000), spin=spin)
    if kind == "frame":
        integrator = rng.choice(("rk4", "dp45", "dp45"))
        precision = rng.choice(("fp64", "mixed"))
        w, h = shape(64, {"rk4": 60000, "dp45": 250000}[integrator] * (1 if precision == "fp64" else 4))
        return dict(kind="frame", integrator=integrator, precision=precision, width=w, height=h,
                    crossings=rng.randint(1, 3), fields=rng.choice(("all", "disk")), sky=rng.random() < 0.5,
                    spin=spin, incl=incl)
    if kind == "closed":
        w, h = shape(64, 3000000)
        return dict(kind="frame", integrator="closed", precision=rng.choice(("fp64", "mixed")), width=w, height=h,
                    crossings=rng.randint(1, 3), fields=rng.choice(("all", "disk")), sky=rng.random() < 0.5,
                    spin=spin, incl=incl)
    if kind == "batch":
        return dict(kind="batch", frames=log_int(2, 64), crossings=rng.randint(1, 3), sky=rng.random() < 0.5)
    if kind == "surrogate":
        w, h = shape(4096, 4000000)
        return dict(kind="surrogate", width=w, height=h, crossings=rng.randint(1, 2),
                    fields=rng.choice(("all", "disk")), spin=spin, incl=incl)
    if kind == "train":
        return dict(kind="train", batch=128 * log_int(1, 128))
    if kind == "forward":
        return dict(kind="forward", rows=log_int(1, 2000000))
    if kind == "transfer":
        precision = rng.choice(("fp64", "mixed"))
        w, h = shape(256, 25600 if precision == "fp64" else 262144)
        return dict(kind="transfer", precision=precision, width=w, height=h, spin=spin, incl=incl)
    w, h = shape(1000, 2000000)
    if kind == "render":
        return dict(kind="render", width=w, height=h, spin=spin, incl=incl, distance=round(rng.uniform(6.0, 30.0), 3))
    return dict(kind="post", width=w, height=h, bloom=round(rng.uniform(0.1, 1.0), 3))


# ---- inputs -------------------------------------------------------------------


def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, 77])


def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _view(case, seed):
    """Spin, inclination [rad] and image-plane window of a frame: the case's, moved a little by the seed."""
    r = _rng(case, seed)
    spin = min(0.998, max(0.0, case["spin"] + float(r.uniform(-0.01, 0.01))))
    incl = math.radians(min(88.5, max(4.5, case["incl"] + float(r.uniform(-0.5, 0.5)))))
    half = 20.0 if case["kind"] == "transfer" else 12.0
    aspect = case["width"] / case["height"]
    dx, dy = (float(v) for v in r.uniform(-0.05, 0.05, 2))
    ha, hb = (half, half / aspect) if aspect >= 1.0 else (half * aspect, half)
    return spin, incl, (-ha + dx, ha + dx), (-hb + dy, hb + dy)


def _scene(case, seed):
    spin, incl, al, be = _view(case, seed)
    kw = dict(width=case["width"], height=case["height"], spin=spin, theta_obs=incl, alpha_min=al[0], alpha_max=al[1],
              beta_min=be[0], beta_max=be[1], precision=int(case.get("precision", "mixed") == "mixed"),
              integrator=INTEGRATORS[case.get("integrator", "dp45")], max_crossings=case.get("crossings", 1))
    if case["kind"] == "transfer":
        kw["max_steps"] = 2000
    return kerr.scene(**kw)


def _batch_views(case, seed):
    r = _rng(case, seed)
    views = []
    for i in range(case["frames"]):
        views.append(dict(side=SIDES[(i * 7 + i // 4) % 4], spin=float(r.uniform(0.0, 0.998)),
                          incl=math.radians(float(r.uniform(5.0, 88.0))),
                          r_obs=float(math.exp(r.uniform(math.log(100.0), math.log(5000.0))))))
    return views


def _ray_inputs(case, seed, device):
    """Start states and constants of ingoing rays in geometric units: theta and q allow the motion."""
    n, g = case["n"], _gen(seed, device)

    def u(lo, hi):
        return lo + (hi - lo) * torch.rand(n, dtype=torch.float64, device=device, generator=g)

    theta = u(0.6, math.pi - 0.6)
    lz = u(-5.0, 5.0)
    q = lz * lz / torch.sin(theta) ** 2 + u(0.5, 20.0)
    state = {"r": u(12.0, 40.0), "theta": theta, "phi": torch.zeros_like(lz), "t": torch.zeros_like(lz),
             "sign_r": torch.full_like(lz, -1.0),
             "sign_theta": torch.where(u(-1.0, 1.0) < 0, -torch.ones_like(lz), torch.ones_like(lz))}
    return state, torch.ones_like(lz), lz, q


GEOM_MASS = 2.99792458e10**2 / 6.67430e-8  # grams with G m / c^2 = 1 cm


def _ray_setup(case):
    return dict(spin=case["spin"], step=4e-4, r_escape=60.0, steps=case["steps"])


def _train_inputs(case, seed, device):
    """Rays over the network's input domain and targets of the tracer's ranges; weights of a fresh network."""
    n, g = case["batch"], _gen(seed, device)

    def u(lo, hi, size=n):
        return lo + (hi - lo) * torch.rand(size, device=device, generator=g)

    x = torch.stack([u(-15.0, 15.0), u(-15.0, 15.0), u(0.0, 0.998), u(0.02, 0.996)], 1)
    cls = torch.randint(0, 3, (n,), device=device, generator=g)
    nc = torch.where(cls == 1, torch.randint(1, 3, (n,), device=device, generator=g), torch.zeros_like(cls))
    t = torch.zeros(n, 16, device=device)
    t[:, 0], t[:, 1] = cls.float(), nc.float()
    one, two, esc = (nc >= 1).float(), (nc >= 2).float(), (cls == 2).float()
    for col, mask in ((2, one), (5, two)):
        ph = u(-math.pi, math.pi)
        t[:, col] = u(-1.2, 1.4) * mask
        t[:, col + 1], t[:, col + 2] = torch.cos(ph) * mask, torch.sin(ph) * mask
    t[:, 8] = u(-0.6, 0.3) * one
    ph = u(-math.pi, math.pi)
    t[:, 9] = u(-1.0, 1.0) * esc
    t[:, 10], t[:, 11] = torch.cos(ph) * esc, torch.sin(ph) * esc
    r = np.random.default_rng([int(seed) & 0x7FFFFFFF, 5])
    p = []
    for k, m in zip(S.LAYER_K, S.LAYER_N):
        used = S.N_FEATURES_USED if k == S.N_FEATURES else k
        w = np.zeros((m, k), np.float32)
        w[:, :used] = r.uniform(-1.0, 1.0, (m, used)) * math.sqrt(3.0 / used)
        p += [w.ravel(), r.uniform(-0.05, 0.05, m).astype(np.float32)]
    return x, t, np.concatenate(p)


def _forward_inputs(case, seed, device):
    n, g = case["rows"], _gen(seed, device)
    lo = torch.tensor([-15.0, -15.0, 0.0, 0.02], device=device)
    hi = torch.tensor([15.0, 15.0, 0.998, 0.996], device=device)
    return lo + (hi - lo) * torch.rand(n, 4, device=device, generator=g)


def _post_input(case, seed, device):
    """A rendered frame's values: mostly dim, a few percent well above the bloom threshold."""
    n = case["width"] * case["height"]
    v = torch.randn(n, 4, device=device, generator=_gen(seed, device)) * 1.2 - 1.5
    fb = torch.exp(v)
    fb[:, 3] = 1.0
    return fb


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rays":
        state, e, lz, q = _ray_inputs(case, seed, "cuda")
        k = _ray_setup(case)
        tracer = kerr.KerrRaytracer(GEOM_MASS, k["spin"])
        tracer.set_step_size(k["step"])
        tracer.set_escape_radius(k["r_escape"])
        tracer.set_max_steps(k["steps"])
        return dict(kind=kind, tracer=tracer, state=state, e=e, lz=lz, q=q)
    if kind in ("frame", "surrogate"):
        scene = _scene(case, seed)
        outs = kerr.alloc_image_outputs(scene, fields=list(DISK_FIELDS if case["fields"] == "disk" else ALL_FIELDS))
        st = dict(kind=kind, scene=scene, outs=outs)
        if kind == "surrogate":
            st["net"] = S.Surrogate(max_batch=128)
            st["net"].load(WEIGHTS)
        else:
            st["sky"] = kerr.sky_generate(512, 10_000, int(seed) & 0xFFFF) if case["sky"] else None
        return st
    if kind == "batch":
        scenes = [kerr.scene(width=v["side"], height=v["side"], spin=v["spin"], theta_obs=v["incl"], r_obs=v["r_obs"],
                             integrator=1, precision=1, max_crossings=case["crossings"])
                  for v in _batch_views(case, seed)]
        # one buffer per field for the whole batch; each frame writes its own slice
        mc, total = case["crossings"], sum(s.width * s.height for s in scenes)
        planes = {f: mc if f in ("r_hit", "phi_hit", "g") else 1 for f in ALL_FIELDS}
        buf = {f: torch.empty(planes[f] * total, dtype=torch.int32 if f in INT_FIELDS else torch.float64,
                              device="cuda") for f in ALL_FIELDS}
        outs, at = [], 0
        for s in scenes:
            n = s.width * s.height
            outs.append({f: buf[f][planes[f] * at:planes[f] * (at + n)] for f in ALL_FIELDS})
            at += n
        b = kerr.TraceBatch(scenes, outs=outs)
        if case["sky"]:
            b.set_sky(kerr.sky_generate(512, 10_000, int(seed) & 0xFFFF))
        return dict(kind=kind, batch=b, buf=buf)
    if kind == "train":
        x, t, params = _train_inputs(case, seed, "cuda")
        net = S.Surrogate(max_batch=case["batch"])
        net.set_params(params)
        return dict(kind=kind, net=net, x=x, t=t)
    if kind == "forward":
        net = S.Surrogate(max_batch=128)
        net.load(WEIGHTS)
        x = _forward_inputs(case, seed, "cuda")
        return dict(kind=kind, net=net, x=x, out=torch.empty(x.shape[0], S.HEAD, device="cuda"))
    if kind == "transfer":
        medium = rt.Medium(torus=rt.torus_defaults(seed=int(seed) & 0xFFFF))
        return dict(kind=kind, scene=_scene(case, seed), medium=medium, lut=rt.Lut(), prm=rt.rt_defaults())
    if kind == "render":
        spin, incl, _, _ = _view(case, seed)
        p = legacy.bridge_params(spin, case["distance"] + float(_rng(case, seed).uniform(-0.1, 0.1)), incl, 1.0,
                                 case["width"], case["height"])
        return dict(kind=kind, params=p, fb=torch.empty(case["width"] * case["height"], 4, device="cuda"))
    if kind == "post":
        src = _post_input(case, seed, "cuda")
        return dict(kind=kind, src=src, fb=torch.empty_like(src), width=case["width"], height=case["height"],
                    bloom=case["bloom"])
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "rays":
        r = state["tracer"].trace(state["state"], state["e"], state["lz"], state["q"])
        return [r.status, r.steps_taken, r.total_distance, r.final_r, r.final_theta, r.final_phi, r.redshift]
    if kind == "frame":
        return kerr.trace_image(state["scene"], state["outs"], sky=state["sky"])
    if kind == "surrogate":
        return state["net"].trace_image(state["scene"], state["outs"])
    if kind == "batch":
        state["batch"].trace()
        return state["buf"]
    if kind == "train":
        return list(state["net"].gradients(state["x"], state["t"]))
    if kind == "forward":
        return state["net"].forward(state["x"], out=state["out"])
    if kind == "transfer":
        return rt.trace(state["scene"], state["medium"], state["lut"], state["prm"])
    if kind == "render":
        legacy.launch(state["params"], state["fb"])
        return state["fb"]
    # a new frame arrives from the renderer each time: the post-processing works in place
    state["fb"].copy_(state["src"])
    legacy.postprocess(state["fb"], state["width"], state["height"], bloom_strength=state["bloom"])
    return state["fb"]


def _out_bytes(n, crossings, fields):
    per = {"cls": 4, "steps": 4, "n_cross": 4}
    return n * sum(per.get(f, 8) * (crossings if f in ("r_hit", "phi_hit", "g") else 1) for f in fields)


def work(case):
    """Bytes: inputs read once, outputs written once. FLOPs: the accepted steps that the scheme and its tolerance
    ask for (per ray about 200 of DP45, 2600 of RK4), or the closed form's evaluations, the network's products."""
    kind = case["kind"]
    if kind == "rays":  # about two thirds of the steps allowed, 4 right-hand sides of about 60 operations each
        return dict(bytes=case["n"] * (9 * 8 + 2 * 4 + 5 * 8), flops=case["n"] * 0.66 * case["steps"] * 260.0)
    if kind == "train":
        n = case["batch"]
        params = sum(k * m + m for k, m in zip(S.LAYER_K, S.LAYER_N))
        return dict(bytes=n * (16 + 64) + 8 * params, flops=3.0 * MLP_FLOPS * n)
    if kind == "forward":
        return dict(bytes=case["rows"] * (16 + 64), flops=MLP_FLOPS * case["rows"])
    if kind == "batch":
        n = sum(SIDES[(i * 7 + i // 4) % 4] ** 2 for i in range(case["frames"]))
        return dict(bytes=_out_bytes(n, case["crossings"], ALL_FIELDS), flops=n * 200 * 506.0)
    n = case["width"] * case["height"]
    if kind == "frame":
        fields = DISK_FIELDS if case["fields"] == "disk" else ALL_FIELDS
        per = {"rk4": 2600 * 213.0, "dp45": 200 * 506.0, "closed": 3000.0}[case["integrator"]]
        return dict(bytes=_out_bytes(n, case["crossings"], fields) + (3145728 if case["sky"] else 0), flops=n * per)
    if kind == "surrogate":
        fields = DISK_FIELDS if case["fields"] == "disk" else ALL_FIELDS
        return dict(bytes=_out_bytes(n, case["crossings"], fields), flops=n * MLP_FLOPS)
    if kind == "transfer":
        return dict(bytes=n * 24 + 128 * 64 * 64 * 16 + 256 * 256 * 4, flops=n * 200 * 1001.0)
    if kind == "render":
        return dict(bytes=n * 16, flops=n * 200 * 506.0)
    return dict(bytes=n * 48, flops=n * 3 * 2 * 2 * 124.0)


# ---- values in 64 bits ----------------------------------------------------------


def _isco(a):
    z1 = 1 + (1 - a * a) ** (1 / 3) * ((1 + a) ** (1 / 3) + (1 - a) ** (1 / 3))
    z2 = math.sqrt(3 * a * a + z1 * z1)
    return 3 + z2 - math.sqrt(max(0.0, (3 - z1) * (3 + z1 + 2 * z2)))


def _taylor(x0, v0, force):
    """Coefficients 0..ORDER of the solution of x'' = force(x) through (x0, v0), force a cubic (c1, c2, c3) in x."""
    c1, c2, c3 = force
    xs, sq = [x0, v0], []
    for k in range(ORDER - 1):
        s = xs[0] * xs[k]
        for i in range(1, k + 1):
            s.addcmul_(xs[i], xs[k - i])
        sq.append(s)
        cube = xs[0] * sq[k]
        for i in range(1, k + 1):
            cube.addcmul_(xs[i], sq[k - i])
        nxt = c1 * xs[k] + c3 * cube
        if c2 is not None:
            nxt.addcmul_(c2, s)
        xs.append(nxt / ((k + 1) * (k + 2)))
    return xs


def _horner(xs, t):
    v = xs[-1].clone()
    for c in reversed(xs[:-1]):
        v = v * t + c
    return v


def _slope(xs, t):
    v = xs[-1] * (len(xs) - 1)
    for k in range(len(xs) - 2, 0, -1):
        v = v * t + k * xs[k]
    return v


ORDER, STEP, MAX_STEPS = 16, 0.004, 2500


def _exact_pixels(a, incl, al, be, width, height, crossings, r_obs=1000.0, device="cuda"):
    """Disk hits of the image-plane rays of one frame, by a Taylor series in Mino time of x = 1/r and u = cos theta:
    x'' and u'' are cubics in x and u (the derivatives of the radial and polar potentials), so the series follows by
    recurrence. The rays' Carter constants are those of the default potentials (q = eta + lambda^2 in both)."""
    f64 = torch.float64
    n = width * height
    i = torch.arange(n, device=device)
    alpha = al[0] + ((i % width).to(f64) + 0.5) * (al[1] - al[0]) / width
    beta = be[0] + ((i // width).to(f64) + 0.5) * (be[1] - be[0]) / height
    so, co = math.sin(incl), math.cos(incl)
    lam = -alpha * so
    q = beta**2 + (alpha**2 - a * a) * co**2 + lam**2
    K = q + (lam - a) ** 2
    r_plus = 1.0 + math.sqrt(1.0 - a * a)
    x_stop, x_esc = 1.0 / (1.001 * r_plus), 1.0 / (1.01 * r_obs)
    r_in, r_out = _isco(a), 30.0
    b = a * a - a * lam  # A = r^2 + b; P(x) = x^4 R = (1 + b x^2)^2 - K x^2 (1 - 2x + a^2 x^2)
    fx = (2 * b - K, 3 * K, 2 * (b * b - K * a * a))
    fu = (a * a - q, None, torch.full_like(q, -2 * a * a))
    x = torch.full_like(q, 1.0 / r_obs)
    P = (1 + b * x**2) ** 2 - K * x**2 * (1 - 2 * x + a * a * x**2)
    vx = P.clamp(min=0).sqrt()
    u = torch.full_like(q, co)
    vu = beta * so
    r_hit = torch.zeros(crossings, n, dtype=f64, device=device)
    hits = torch.zeros(n, dtype=torch.long, device=device)
    at = i
    for _ in range(MAX_STEPS):
        tx, tu = _taylor(x, vx, fx), _taylor(u, vu, fu)
        x1, u1 = _horner(tx, STEP), _horner(tu, STEP)
        cross = (u * u1 < 0).nonzero().squeeze(1)
        if cross.numel():
            cu, cx = [c[cross] for c in tu], [c[cross] for c in tx]
            t = STEP * u[cross] / (u[cross] - u1[cross])
            for _ in range(5):
                t = (t - _horner(cu, t) / _slope(cu, t)).clamp(0.0, STEP)
            xc = _horner(cx, t)
            r = 1.0 / xc
            ok = (xc > 0) & (xc < x_stop) & (r >= r_in) & (r <= r_out)
            p = at[cross][ok]
            r_hit[hits[p], p] = r[ok]
            hits[p] += 1
        vx, vu, x, u = _slope(tx, STEP), _slope(tu, STEP), x1, u1
        live = ((hits[at] < crossings) & (x < x_stop) & ((x > x_esc) | (vx > 0))).nonzero().squeeze(1)
        if not live.numel():
            break
        if live.numel() < at.numel():
            at, x, vx, u, vu = at[live], x[live], vx[live], u[live], vu[live]
            fx = tuple(c[live] for c in fx)
            fu = (fu[0][live], None, fu[2][live])
    r = torch.where(r_hit > 0, r_hit, torch.full_like(r_hit, 10.0))
    s = r.sqrt() ** 3
    g = (s * (s - 3 * r.sqrt() + 2 * a)).clamp(min=0).sqrt() / (s + a - lam)
    g = torch.where(r_hit > 0, g, torch.zeros_like(g))
    peak = (1 - math.sqrt(1 / 1.5)) / (1.5 * r_in) ** 3
    flux = ((1 - (r_in / r[0]).sqrt()).clamp(min=0) / r[0] ** 3 / peak).clamp(max=1.0)
    flux = torch.where(r_hit[0] > 0, flux, torch.zeros_like(flux))
    intensity = (g**4 * (r_in / r) ** 3 * (r_hit > 0)).sum(0)
    return dict(r_hit=r_hit, g=g, flux=flux, intensity=intensity)


def _exact_frame(case, seed):
    spin, incl, al, be = _view(case, seed)
    v = _exact_pixels(spin, incl, al, be, case["width"], case["height"], case["crossings"])
    if case.get("sky"):
        v["intensity"] = None  # the sky's texel goes into it
    # the azimuths and the escape direction depend on where a stepper's last step ends
    return {f: v.get(f) for f in (DISK_FIELDS if case["fields"] == "disk" else ALL_FIELDS)}


def _exact_batch(case, seed):
    out = {f: [] for f in ("r_hit", "g", "flux", "intensity")}
    for w in _batch_views(case, seed):
        v = _exact_pixels(w["spin"], w["incl"], (-12.0, 12.0), (-12.0, 12.0), w["side"], w["side"], case["crossings"],
                          w["r_obs"])
        for f in out:
            out[f].append(v[f].reshape(-1))
    done = {f: torch.cat(v) for f, v in out.items()}
    if case["sky"]:
        done["intensity"] = None
    return {f: done.get(f) for f in ALL_FIELDS}


def _exact_rays(case, seed):
    """The first-order scheme of the batched API (RK4 in Mino time with sign flips), in 64 bits."""
    st, e, lz, q = _ray_inputs(case, seed, "cuda")
    k = _ray_setup(case)
    a, h = k["spin"], k["step"]
    r_stop = 1.001 * (1.0 + math.sqrt(1.0 - a * a))
    y = torch.stack([st["r"], st["theta"], st["phi"]])
    sr, sth = st["sign_r"].clone(), st["sign_theta"].clone()
    steps = torch.zeros_like(lz)

    def pots(y):
        sin2 = torch.sin(y[1]).square().clamp(min=1e-12)
        delta = y[0] ** 2 - 2.0 * y[0] + a * a
        A = (y[0] ** 2 + a * a) - a * lz
        R = A * A - delta * (q + (lz - a) ** 2)
        Th = q + a * a * torch.cos(y[1]) ** 2 - lz * lz / sin2
        return R, Th, sin2, delta, A

    def deriv(y):
        R, Th, sin2, delta, A = pots(y)
        return torch.stack([sr * R.clamp(min=0).sqrt(), sth * Th.clamp(min=0).sqrt(),
                            lz / sin2 - a + a * A / delta.clamp(min=1e-12)])

    for _ in range(k["steps"]):
        live = (y[0] > r_stop) & (y[0] < k["r_escape"])
        R, Th = pots(y)[:2]
        sr = torch.where(live & (R < 0), -sr, sr)
        sth = torch.where(live & (Th < 0), -sth, sth)
        k1 = deriv(y)
        k2 = deriv(y + 0.5 * h * k1)
        k3 = deriv(y + 0.5 * h * k2)
        k4 = deriv(y + h * k3)
        z = y + h * (k1 + 2 * k2 + 2 * k3 + k4) / 6.0
        z[1] = z[1].clamp(1e-6, math.pi - 1e-6)
        y = torch.where(live, z, y)
        steps += live.double()
    return [None, None, steps * h, y[0], y[1], y[2], None]


def _features(x):
    x = x.double()
    sc = torch.stack([x[:, 0] / 15, x[:, 1] / 15, 2 * x[:, 2] - 1, 2 * x[:, 3] - 1], 1)
    lam = -x[:, 0] * (1 - x[:, 3] ** 2).clamp(min=0).sqrt() / 15
    eta = (x[:, 1] ** 2 + (x[:, 0] ** 2 - x[:, 2] ** 2) * x[:, 3] ** 2) / 225
    freq = math.pi * 2.0 ** (torch.arange(16, device=x.device, dtype=torch.float64) / 3)
    ang = sc[:, :, None] * freq
    four = torch.stack([torch.sin(ang), torch.cos(ang)], 3).reshape(x.shape[0], 128)
    return torch.cat([four, sc, lam[:, None], eta[:, None]], 1)


def _head(x, p):
    h, off = _features(x), 0
    for k, m in zip(S.LAYER_K, S.LAYER_N):
        w, b = p[off:off + m * k].view(m, k), p[off + m * k:off + m * k + m]
        off += m * k + m
        h = h @ w[:, :h.shape[1]].T + b
        if m == S.HIDDEN:
            h = torch.nn.functional.silu(h)
    return h


def _exact_train(case, seed):
    x, t, params = _train_inputs(case, seed, "cuda")
    p = torch.from_numpy(params).cuda().double().requires_grad_()
    o, t = _head(x, p), t.double()
    cls, nc = t[:, 0].long(), t[:, 1]
    ce = torch.nn.functional.cross_entropy(o[:, :3], cls, reduction="sum")
    one, two, esc = nc >= 1, nc >= 2, cls == 2
    mask = torch.stack([one, one, one, two, two, two, one, esc, esc, esc], 1)
    sq = (((o[:, 3:13] - t[:, 2:12]) ** 2) * mask).sum()
    ((ce + sq) / x.shape[0]).backward()
    return [p.grad, None]  # the sums of the loss are FP32 atomics over classes: counts among them


def _exact_forward(case, seed):
    p = torch.from_numpy(np.load(WEIGHTS)["params"]).cuda().double()
    x = _forward_inputs(case, seed, "cuda")
    return torch.cat([_head(v, p) for v in x.split(1 << 18)])


def _exact_post(case, seed):
    w, h = case["width"], case["height"]
    c = _post_input(case, seed, "cuda")[:, :3].double().view(h, w, 3)
    lum = (c * torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=c.device)).sum(2)
    bright = c * torch.where(lum > 0.001, (lum - 1.0).clamp(min=0) / lum, torch.zeros_like(lum))[:, :, None]
    bright = bright.permute(2, 0, 1)[:, None]
    bloom = torch.zeros_like(bright)
    for r in (4, 8, 16, 32):
        k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=c.device, dtype=torch.float64) / (r / 2)) ** 2)
        k = k / k.sum()
        v = torch.nn.functional.pad(bright, (r, r, r, r), mode="replicate") if r < min(w, h) else None
        if v is None:  # replicate padding wider than the image
            ys = torch.arange(-r, h + r, device=c.device).clamp(0, h - 1)
            xs = torch.arange(-r, w + r, device=c.device).clamp(0, w - 1)
            v = bright[:, :, ys][:, :, :, xs]
        for i in range(2 * r + 1):  # one axis, then the other
            t = k[i] * v[:, :, :, i:i + w]
            rows = t if i == 0 else rows + t
        for i in range(2 * r + 1):
            bloom = bloom + k[i] * rows[:, :, i:i + h]
    col = c + case["bloom"] * bloom[:, 0].permute(1, 2, 0)
    # uv and the index int(u w), int(v h) are FP32 by definition (numpy: correctly rounded quotients)
    px, py = np.arange(w, dtype=np.float32) / np.float32(w), np.arange(h, dtype=np.float32) / np.float32(h)
    rx = torch.from_numpy((px * np.float32(w)).astype(np.int64)).to(c.device).clamp(0, w - 1)
    ry = torch.from_numpy((py * np.float32(h)).astype(np.int64)).to(c.device).clamp(0, h - 1)
    u, v = torch.from_numpy(px).to(c.device), torch.from_numpy(py).to(c.device)
    moved = col[ry][:, rx]  # red and blue are looked up at int(u w), int(v h)
    d2 = (u.double() - 0.5)[None, :] ** 2 + (v.double() - 0.5)[:, None] ** 2
    vig = (1 - 0.5 * d2).clamp(min=0).sqrt()
    z = torch.stack([moved[:, :, 0], col[:, :, 1], moved[:, :, 2]], 2) * 12.0 * vig[:, :, None]
    z = ((z * (2.51 * z + 0.03)) / (z * (2.43 * z + 0.59) + 0.14)).clamp(0, 1) ** (1 / 2.2)
    return torch.cat([z, torch.ones_like(z[:, :, :1])], 2).view(w * h, 4)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("frame", "surrogate"):
        return _exact_frame(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "rays":
        return _exact_rays(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "forward":
        return _exact_forward(case, seed)
    if kind == "post":
        return _exact_post(case, seed)
    # transfer: the medium is sampled along the integrator's own steps; render: an art-directed look
    return None
