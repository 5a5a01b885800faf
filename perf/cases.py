"""The calls that users of the engine make, as timed cases.

A case is one call (or, for a movie frame, one upload and one render) through
raptor_gb300.engine: renders and VJPs in the three arithmetic forms, both
cameras and integrators, one to five frequencies, from the 12x12 smoke image
to the 1024x1024 benchmark image.  The dumps are the seeded synthetic torus of
raptor_gb300.synth.  The FP64 form's results are returned as they come
(float64); the mixed forms compute their transfer in FP32, and a caller keeps
their images (in janskys, as the host program writes them: in cgs units the
log-polar camera's are below float32's range) and gradients in float32.

Linear images have even widths, log-polar ones odd heights: else a line of
pixels looks exactly down the polar axis, where rays amplify a rounding of
their state 1e8 times and no two orders of the same operations agree.

exact() restates the imaging path in plain torch float64: the same pixels,
steps and samples, gradients by automatic differentiation.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from raptor_gb300 import engine, synth

FORMS = {"fp64": engine.PREC_FP64, "mixed": engine.PREC_MIXED, "mixed_df": engine.PREC_MIXED_DF}
FIVE = (86e9, 150e9, 230e9, 345e9, 690e9)
JANSKY = 1e23  # per cgs unit of flux density
BATCH_FREQS = (86e9, 230e9, 345e9)
FIELDS = ("d_rho", "d_u", "d_lnthetae")
SCALARS = ("d_m_unit", "d_r_high", "d_r_low", "d_inclination")


def _freqs(n):
    return (230e9,) if n == 1 else FIVE[:n]


def listed():
    render = dict(op="render", camera="linear", integrator="rk4", n_freq=1, incl=60.0, spin=0.9375)
    return [
        # a single thumbnail, the smoke test's render: launches and one ray's latency
        dict(render, name="thumbnail_fp64", form="fp64", width=12, height=12, grid=64),
        # a preview at the size the reference ships its image with
        dict(render, name="preview_fp64", form="fp64", width=100, height=100, grid=256),
        # the benchmark image, in each arithmetic form
        dict(render, name="image_fp64", form="fp64", width=1024, height=1024, grid=512),
        dict(render, name="image_mixed", form="mixed", width=1024, height=1024, grid=512),
        dict(render, name="image_mixed_df", form="mixed_df", width=1024, height=1024, grid=512),
        # a spectrum of images, odd sizes, nearly face-on
        dict(render, name="spectral_fp64", form="fp64", width=334, height=251, grid=256, n_freq=5, incl=17.0),
        # a parameter survey: images of uneven sizes over two dumps in one launch
        dict(op="batch", name="survey_fp64", form="fp64", small=12, middle=6, large=1, grid=256),
        # one gradient of a fit to an observed image
        dict(render, op="vjp", name="gradient_fp64", form="fp64", width=128, height=128, grid=256),
        # gradients of a fit at five frequencies, in the forms a fit's inner loop takes
        dict(render, op="vjp", name="gradient_mixed", form="mixed", width=512, height=512, grid=512, n_freq=5),
        dict(render, op="vjp", name="gradient_mixed_df", form="mixed_df", width=512, height=512, grid=512, n_freq=5),
        # a movie frame: a new dump goes up, one image comes back
        dict(render, op="frame", name="frame_mixed_df", form="mixed_df", width=256, height=256, grid=512),
        # the log-polar camera with the midpoint integrator
        dict(render, name="logcam_mixed", form="mixed", width=151, height=97, grid=256, n_freq=2, camera="log",
             integrator="rk2"),
    ]


# pixels of one render or VJP that cost about what the largest listed case does
_MOST = {"fp64": 7e5, "mixed": 8e5, "mixed_df": 1.2e6}


def draw(rng):
    op = rng.choice(["render", "render", "render", "vjp", "vjp", "frame", "batch"])
    form = rng.choice(list(FORMS))
    grid = rng.choice([64, 128, 256, 512])
    if op == "batch":
        return dict(op="batch", form=form, small=rng.randint(2, 16), middle=rng.randint(1, 6), large=rng.randint(0, 1),
                    grid=min(grid, 256))
    n_freq = rng.choice([1, 1, 2, 3, 5, 8]) if op != "vjp" else rng.choice([1, 2, 5])
    most = _MOST[form] / (1.0 + 0.1 * n_freq) / (4.0 if op == "vjp" else 1.0)
    pixels = math.exp(rng.uniform(math.log(64.0), math.log(most)))
    aspect = math.exp(rng.uniform(-0.7, 0.7))
    width = max(8, min(2048, round(math.sqrt(pixels * aspect))))
    height = max(8, min(2048, round(pixels / width)))
    camera = rng.choice(["linear", "linear", "log"])
    if camera == "log":
        height |= 1
    else:
        width += width % 2
    return dict(op=op, form=form, width=width, height=height, grid=grid, n_freq=n_freq,
                incl=rng.uniform(8.0, 172.0), spin=rng.choice([0.8, 0.9, 0.9375]),
                camera=camera, integrator=rng.choice(["rk4", "rk4", "rk4", "rk2"]))


@functools.lru_cache(maxsize=8)
def _torus(n, spin):
    return synth.make_torus(n1=n, n2=n, a=spin, noise=0.0)


def _dump(case, seed, spin):
    """Geometry and primitives: the torus with a seeded log-normal perturbation of rho and u."""
    d = _torus(case["grid"], spin)
    prims = d.prims.copy()
    rng = np.random.default_rng([seed, int(spin * 1e4)])
    prims[:2] *= np.exp(0.04 * rng.standard_normal(prims[:2].shape))
    return d.geom, prims


def _inputs(case, seed):
    """Dumps, image descriptions (as plain keywords) and loss weights of a case."""
    rng = np.random.default_rng([seed, 7])
    if case["op"] == "batch":
        dumps = [_dump(case, seed, s) for s in (0.5, 0.9375)]
        images = [dict(width=n, height=n, freqs=(float(rng.choice(BATCH_FREQS)),), grid=int(rng.integers(2)),
                       inclination=float(rng.uniform(5.0, 175.0)), m_unit=float(10 ** rng.uniform(18.0, 20.0)))
                  for n in [128] * case["small"] + [256] * case["middle"] + [512] * case["large"]]
        return dumps, images, None
    dumps = [_dump(case, seed, case["spin"])]
    n_freq = case["n_freq"]
    freqs = _freqs(n_freq) if n_freq <= 5 else tuple(FIVE) + tuple(1e11 * k for k in range(1, n_freq - 4))
    image = dict(width=case["width"], height=case["height"], freqs=freqs, grid=0,
                 inclination=case["incl"] + float(rng.uniform(-0.5, 0.5)), m_unit=float(10 ** rng.uniform(18.9, 19.1)),
                 integrator=engine.RK2 if case["integrator"] == "rk2" else engine.RK4,
                 camera=engine.CAM_LOG if case["camera"] == "log" else engine.CAM_LINEAR)
    weights = None
    if case["op"] == "vjp":
        weights = 1.0 + 0.3 * rng.standard_normal(case["width"] * case["height"] * n_freq)
        if case["camera"] == "log":
            weights *= 1e20  # an image in flux units: the loss is in units of the observation's error
    return dumps, [image], weights


def prepare(case, seed):
    """A context with the dumps on the device, the image descriptions and the loss weights."""
    dumps, images, weights = _inputs(case, seed)
    eng = engine.Engine(use_graph=1 if case["op"] == "batch" else 0)
    ids = [eng.upload_grid(geom, prims) for geom, prims in dumps]
    descs = [engine.image_desc(**dict(im, grid=ids[im["grid"]])) for im in images]
    return dict(op=case["op"], form=case["form"], eng=eng, ids=ids, dumps=dumps, descs=descs, weights=weights)


def _kept(out, form):
    if form == "fp64":
        return out
    return {k: (v * JANSKY if k in ("image", "spectrum") else v).astype(np.float32) for k, v in out.items()}


def run(state):
    eng, form = state["eng"], FORMS[state["form"]]
    if state["op"] == "frame":
        geom, prims = state["dumps"][0]
        eng.upload_grid(geom, prims, state["ids"][0])
    if state["op"] == "vjp":
        image, grad = eng.vjp(state["descs"][0], state["weights"], form)
        out = dict(image=image, **{k: np.asarray(grad[k]) for k in SCALARS + FIELDS})
    else:
        image, spectrum = eng.render(state["descs"], form)
        out = dict(image=image, spectrum=spectrum)
    return _kept(out, state["form"])


# Operations of the path per unit of work (the imaging algorithm's own count:
# each +, -, *, / and library call is one), and about how many units a ray
# takes: the step count follows from the step-size rule, the samples from the
# share of a ray's steps inside the grid.
_STEP = {"rk4": 1648, "rk2": 814}
_STEPS_A_RAY, _SAMPLES_A_RAY = 280, 155


def work(case):
    if case["op"] == "batch":
        sizes = [(128, case["small"]), (256, case["middle"]), (512, case["large"])]
        rays = sum(n * n * k for n, k in sizes)
        outputs, n_freq, step, grids, adjoint = rays, 1, _STEP["rk4"], 2, False
    else:
        rays, n_freq = case["width"] * case["height"], case["n_freq"]
        outputs, step, grids, adjoint = rays * n_freq, _STEP[case["integrator"]], 1, case["op"] == "vjp"
    cells = case["grid"] ** 2
    size = 4 if case["form"] != "fp64" else 8
    nbytes = 8 * size * cells * grids + 8 * outputs
    if case["op"] == "frame":
        nbytes += 64 * cells
    if adjoint:
        nbytes += 8 * outputs + 3 * 8 * cells
    flops = rays * (138 + step * _STEPS_A_RAY + (388 + 109 * n_freq) * _SAMPLES_A_RAY)
    return dict(bytes=nbytes, flops=flops * (2 if adjoint else 1))


# ------------------------------------------------------------------ exact()
R_CAM = 1.0e4
E_CHARGE, E_MASS, P_MASS = 4.8032068e-10, 9.1093826e-28, 1.67262171e-24
BOLTZMANN, LIGHT, PLANCK, GRAVITY = 1.3806505e-16, 2.99792458e10, 6.6260693e-27, 6.6742e-8
E2C, E2CH = 7.695589048e-30, 1.161410e-03
M_BH, SOURCE_DIST, CAM_SIZE, EPS, R_RATIO = 8.9505e39, 2.6228263e22, 40.0, 0.05, 3.0


def _point(x1, x2, h):
    r, sin2 = torch.exp(x1), torch.sin(2 * math.pi * x2)
    theta = math.pi * x2 + 0.5 * (1 - h) * sin2
    dtheta = math.pi * (1 + (1 - h) * torch.cos(2 * math.pi * x2))
    return r, sin2, torch.sin(theta), torch.cos(theta), dtheta


def _rhs(y, a, h):
    """Geodesic equation in MKS coordinates, y = (x1, x2, k^0 .. k^3).  With lengths in units of r
    (w = 1/r, K1 = r k^1, K2 = r^2 k^2, K3 = r^2 k^3) the Kerr-Schild connection has no large factors."""
    x1, x2, k0, k1, k2, k3 = y
    r, sin2, s, c, dth = _point(x1, x2, h)
    w, idth = 1 / r, 1 / dth
    K1, K2, K3 = r * k1, r * r * k2, r * r * k3
    w2, s2, sc, cot = w * w, s * s, s * c, c / s
    sig = 1 + a * a * c * c * w2
    rho = 1 + a * a * w2
    dlt = rho - 2 * w
    i1 = 1 / sig
    i2 = i1 * i1
    i3 = i2 * i1
    be = (2 - sig) * i3
    P = a * s2 * w2 * K3
    ga = i1 - a * a * s2 * be * w2 * w
    X0, X1, Q, H = k0 * (k0 - 2 * P), 2 * K1 * (k0 - P), K1 * K1, (k0 + K1) ** 2
    m = w2 * (i1 * dth * dth * K2 * K2 + ga * s2 * K3 * K3)
    bw, t = be * w, a * a * sc * dth * i1 * w2
    A0 = w * (2 * w * m + 4 * t * i1 * w2 * K2 * (k0 + K1 - P)
              - bw * (2 * w * X0 + (sig + 2 * w) * X1 + 2 * (sig + w) * Q))
    A1 = w2 * (dlt * m + 2 * t * w * K1 * K2 - Q - 2 * i1 * K1 * P
               - bw * (dlt * X0 + (dlt - sig) * X1 - (2 * sig - dlt) * Q))
    A2 = w2 * w * ((t + 2 * math.pi ** 2 * (1 - h) * sin2 * idth) * w * K2 * K2 - 2 * i1 * K1 * K2
                   - sc * i3 * idth * w * (2 * a * K3 * (2 * rho * w * k0 + (sig * sig + 2 * w * rho) * K1)
                                           - (dlt * sig * sig + 2 * w * rho * rho) * K3 * K3 - 2 * a * a * w * H))
    A3 = w2 * w * (2 * a * cot * dth * i2 * w * K2 * (2 * w * k0 + (sig + 2 * w) * K1) - a * bw * (H - 2 * k0 * P)
                   - ga * K3 * (2 * K1 - P) + a * i1 * dth * dth * w2 * K2 * K2
                   - 2 * (cot * dth + 2 * t * i1 * w) * w * K2 * K3)
    return k1, k2, A0, A1, A2, A3


def _advance(y, a, h, rk4):
    """One step of the adaptive integrator, backward in the affine parameter; the step taken."""
    m2 = torch.minimum(y[1], 1 - y[1])
    dl = -torch.clamp(EPS / (y[3].abs() + y[4].abs() / m2 + y[5].abs() + 1e-40), min=1e-12)
    f1 = _rhs(y, a, h)
    f2 = _rhs([p + 0.5 * dl * q for p, q in zip(y, f1)], a, h)
    if not rk4:
        return [p + dl * q for p, q in zip(y, f2)], dl
    f3 = _rhs([p + 0.5 * dl * q for p, q in zip(y, f2)], a, h)
    f4 = _rhs([p + dl * q for p, q in zip(y, f3)], a, h)
    return [p + dl / 6 * (q1 + 2 * q2 + 2 * q3 + q4) for p, q1, q2, q3, q4 in zip(y, f1, f2, f3, f4)], dl


def _cell(x, start, dx, n):
    t = (x - start) / dx - 0.5
    i = t.detach().to(torch.int64)
    d = torch.where(i > n - 2, torch.ones_like(t), torch.where(t < 0, torch.zeros_like(t), t - i))
    return i.clamp(0, n - 2), d


def _lower(g, v):
    g00, g01, g03, g11, g13, g22, g33 = g
    return (g00 * v[0] + g01 * v[1] + g03 * v[3], g01 * v[0] + g11 * v[1] + g13 * v[3], g22 * v[2],
            g03 * v[0] + g13 * v[1] + g33 * v[3])


def _dot(u, v):
    return u[0] * v[0] + u[1] * v[1] + u[2] * v[2] + u[3] * v[3]


def _transfer(y, dl, tau, I, inside, sc):
    """One step of the radiative transfer for the rays that are `inside` the grid."""
    geom, cells, freqs = sc["geom"], sc["cells"], sc["freqs"]
    a, r_high, r_low = geom.a, sc["r_high"], sc["r_low"]
    r, _, s, c, dth = _point(y[0], y[1], geom.hslope)
    s2, i_rho2 = s * s, 1 / (r * r + a * a * c * c)
    z = 2 * r * i_rho2
    g = (z - 1, z * r, -a * z * s2, (1 + z) * r * r, -a * s2 * (1 + z) * r, dth * dth / i_rho2,
         s2 * (1 / i_rho2 + a * a * s2 * (1 + z)))
    u00, u01, u02, u03 = -1 - z, 2 * i_rho2, 0.0, 0.0
    i, d1 = _cell(y[0], geom.startx1, geom.dx1, geom.n1)
    j, d2 = _cell(y[1], geom.startx2, geom.dx2, geom.n2)
    at = i * geom.n2 + j
    v = sum(wt[:, None] * cells[at + o] for wt, o in
            (((1 - d1) * (1 - d2), 0), ((1 - d1) * d2, 1), (d1 * (1 - d2), geom.n2), (d1 * d2, geom.n2 + 1)))
    den, ie, V, Bp, lnf = v[:, 0], v[:, 1], v[:, 2:5].T, v[:, 5:8].T, v[:, 8]
    VV = (g[3] * V[0] + 2 * g[4] * V[2]) * V[0] + g[5] * V[1] * V[1] + g[6] * V[2] * V[2]
    vf = torch.sqrt((1 + VV.abs()) / -u00)
    U = (-vf * u00, V[0] - vf * u01, V[1] - vf * u02, V[2] - vf * u03)
    Uc = _lower(g, U)
    UB = Uc[1] * Bp[0] + Uc[2] * Bp[1] + Uc[3] * Bp[2]
    b = (UB, (Bp[0] + U[1] * UB) / U[0], (Bp[1] + U[2] * UB) / U[0], (Bp[2] + U[3] * UB) / U[0])
    bsq = _dot(b, _lower(g, b))
    lit = inside & (bsq > 0)  # elsewhere any state without singular derivatives: it is not used
    bsq = torch.where(lit, bsq, torch.ones_like(bsq))
    B = torch.sqrt(bsq) * sc["B_unit"] + 1e-20
    beta2 = (ie * (2 / 3) / (bsq + 1e-20)) ** 2
    ratio = (r_high * beta2 + r_low) / (1 + beta2)
    gam = 0.5 * (1 + 2 / 3 * (ratio + 1) / (ratio + 2) + 4 / 3)
    thetae = ie / den * (gam - 1) * (P_MASS / E_MASS) / (1 + ratio) * torch.exp(lnf)
    k = _lower(g, y[2:])
    kU = _dot(k, U)
    cosp = (_dot(k, b) / (kU.abs() * B / sc["B_unit"])).clamp(-1, 1)
    sinp = torch.sqrt((1 - cosp * cosp).clamp(min=1e-30))
    ok = lit & (bsq / den <= 1) & (thetae > 1e-4) & (sinp.abs() >= 1e-10)
    thetae = torch.where(ok, thetae, torch.ones_like(thetae))
    taus, Is = [], []
    for f, nu in enumerate(freqs):
        nu_p = -kU * nu
        nu_s = (2 / 9) * E_CHARGE * B / (2 * math.pi * E_MASS * LIGHT) * thetae * thetae * sinp
        go = ok & (nu_p > 0) & (nu_p < 1e12 * nu_s)  # beyond, exp(-X^1/3) is 0
        nu_p = torch.where(go, nu_p, torch.full_like(nu_p, nu))
        X6 = torch.where(go, nu_p / nu_s, torch.ones_like(nu_p)) ** (1 / 6)
        F = (X6 ** 3 + 2 ** (11 / 12) * X6) ** 2 * torch.exp(-X6 * X6)
        em = den * sc["Ne_unit"] * math.sqrt(2) * math.pi * nu_s / (6 * thetae * thetae) * F
        x = PLANCK * nu_p / (E_MASS * LIGHT * LIGHT * thetae)
        ab = em * E2CH * LIGHT * LIGHT * torch.expm1(torch.where(go, x, torch.ones_like(x))) / (2 * nu_p ** 3)
        path = dl * sc["Rg"] / nu
        t = tau[f] + torch.where(go, nu_p * ab * path, torch.zeros_like(path))
        dI = em * E2C / nu_p ** 2 * torch.exp(-t) * path
        taus.append(t)
        Is.append(I[f] + torch.where(go & (t < math.log(1000.0)) & (t >= 0), dI, torch.zeros_like(dI)))
    return taus, Is


def _camera(im, geom, incl, dev):
    """Initial photons (x1, x2, k^0 .. k^3) of all pixels and the factor from I to the image."""
    a, W, H = geom.a, im["width"], im["height"]
    px = torch.arange(W, device=dev, dtype=torch.float64).repeat(H)
    py = torch.arange(H, device=dev, dtype=torch.float64).repeat_interleave(W)
    rg = GRAVITY * M_BH / LIGHT / LIGHT
    scale = torch.ones_like(px)
    if im.get("camera") == engine.CAM_LOG:
        ri = torch.exp(math.log(20.0) * (px + 0.5) / W) - 1
        th = 2 * math.pi * (py + 0.5) / H
        alpha, beta = ri * torch.cos(th), ri * torch.sin(th)
        scale = ri * (rg * (ri + 1) * math.log(20.0) / W) * (rg * 2 * math.pi / H) / SOURCE_DIST ** 2
    else:
        alpha = -CAM_SIZE * 0.5 + (px + 0.5) * (CAM_SIZE / W)
        beta = -CAM_SIZE * 0.5 + (py + 0.5) * (CAM_SIZE / H)
    mu, st, r = torch.cos(incl * math.pi / 180), torch.sin(incl * math.pi / 180), R_CAM
    lz = -alpha * st
    q = beta * beta + mu * mu * (alpha * alpha - 1)
    kth = torch.sign(beta) * torch.sqrt((q - lz * lz * mu * mu / (st * st) + mu * mu).abs())
    sg, dl = r * r + a * a * mu * mu, r * r + a * a - 2 * r
    A = (r * r + a * a) ** 2 - dl * a * a * st * st
    g00, g03, g33 = -A / (sg * dl), -2 * a * r / (sg * dl), (dl - a * a * st * st) / (sg * dl * st * st)
    u0, u3, u2 = -g00 + g03 * lz, g33 * lz - g03, kth / sg
    u1 = torch.sqrt((u0 - u2 * kth - u3 * lz) * dl / sg) / r
    theta = torch.acos(mu)
    with torch.no_grad():
        x2 = theta / math.pi
        for _ in range(60):
            x2 = x2 - (math.pi * x2 + 0.5 * (1 - geom.hslope) * torch.sin(2 * math.pi * x2) - theta) / (
                math.pi * (1 + (1 - geom.hslope) * torch.cos(2 * math.pi * x2)))
    dth = math.pi * (1 + (1 - geom.hslope) * torch.cos(2 * math.pi * x2))
    x2 = x2 + (theta - theta.detach()) / dth  # the root's dependence on the inclination
    dth = math.pi * (1 + (1 - geom.hslope) * torch.cos(2 * math.pi * x2))
    y = [torch.full_like(px, math.log(r)), torch.zeros_like(px) + x2, u0 + 2 * r / dl * r * u1, u1, u2 / dth,
         a / dl * r * u1 + u3]
    return y, scale


def _image(im, dump, dev, par, cells, checkpoint=None):
    """Image [pixels, frequencies] in float64, differentiable in par and cells."""
    geom = dump[0]
    rg = GRAVITY * M_BH / LIGHT / LIGHT
    rho_unit = par["m_unit"] / (GRAVITY * M_BH / LIGHT ** 2) ** 3
    sc = dict(geom=geom, cells=cells, freqs=im["freqs"], Rg=rg, B_unit=LIGHT * torch.sqrt(4 * math.pi * rho_unit),
              Ne_unit=rho_unit / (P_MASS + E_MASS), r_high=par["r_high"], r_low=par["r_low"])
    y, scale = _camera(im, geom, par["inclination"], dev)
    nf, rk4 = len(im["freqs"]), im.get("integrator") != engine.RK2
    n = y[0].numel()
    lost, stop1, stop2 = (1 + math.sqrt(1 - geom.a ** 2)) * 1.1, geom.stopx1, geom.stopx2
    tau, I = [torch.zeros_like(y[0]) for _ in range(nf)], [torch.zeros_like(y[0]) for _ in range(nf)]
    ids, ended, image = torch.arange(n, device=dev), [], []

    def step(alive, *v):
        y, tau, I = list(v[:6]), list(v[6:6 + nf]), list(v[6 + nf:])
        new, dl = _advance(y, geom.a, geom.hslope, rk4)
        new = [torch.where(alive, p, q) for p, q in zip(new, y)]
        away = (new[0] > stop1) & (new[3] < 0)
        inside = alive & ~away & (new[0] < stop1) & (new[0] > geom.startx1) & (new[1] > geom.startx2) & (new[1] < stop2)
        tau, I = _transfer(new, dl.abs(), tau, I, inside, sc)
        return (*new, *tau, *I)

    alive = torch.ones_like(ids, dtype=torch.bool)
    for count in range(100000):
        if count % 16 == 0 and not bool(alive.all()):
            keep, over = alive.nonzero()[:, 0], (~alive).nonzero()[:, 0]
            ended.append(ids[over])
            image.append(torch.stack([v[over] for v in I], 1))
            ids, y, tau, I = ids[keep], [v[keep] for v in y], [v[keep] for v in tau], [v[keep] for v in I]
            alive = alive[keep]
            if not len(ids):
                break
        out = step(alive, *y, *tau, *I) if checkpoint is None else checkpoint(step, alive, *y, *tau, *I,
                                                                             use_reentrant=False)
        y, tau, I = list(out[:6]), list(out[6:6 + nf]), list(out[6 + nf:])
        r = torch.exp(y[0].detach())
        alive = alive & (r < R_CAM * 1.01) & (r > lost) & ~((y[0] > stop1) & (y[3] < 0))
    flat = torch.zeros(n, nf, dtype=torch.float64, device=dev).index_copy(0, torch.cat(ended), torch.cat(image))
    nu3 = torch.tensor([nu ** 3 for nu in im["freqs"]], dtype=torch.float64, device=dev)
    return flat * nu3 * scale[:, None]


def exact(case, seed):
    adjoint = case["op"] == "vjp"
    if case["op"] == "batch" or (adjoint and case["width"] * case["height"] * case["n_freq"] > 2e4):
        return None  # image after image, or step after step backward: minutes
    if case["width"] * case["height"] * (1 + 0.3 * case["n_freq"]) > 1.5e6:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dumps, (im,), weights = _inputs(case, seed)
    geom, prims = dumps[0]
    f64 = functools.partial(torch.tensor, dtype=torch.float64, device=dev, requires_grad=adjoint)
    par = dict(m_unit=f64(im["m_unit"]), r_high=f64(R_RATIO), r_low=f64(R_RATIO), inclination=f64(im["inclination"]))
    cells = torch.zeros(geom.n1 * geom.n2, 9, dtype=torch.float64, device=dev)
    cells[:, :8] = torch.from_numpy(prims.reshape(8, -1).T.copy()).to(dev)
    cells.requires_grad_(adjoint)
    if not adjoint:
        with torch.no_grad():
            image = _image(im, dumps[0], dev, par, cells)
        return _exact_kept(dict(image=image.reshape(-1).cpu().numpy(), spectrum=image.sum(0).cpu().numpy()), case)
    from torch.utils.checkpoint import checkpoint
    image = _image(im, dumps[0], dev, par, cells, checkpoint)
    loss = (image.reshape(-1) * torch.from_numpy(weights).to(dev)).sum()
    got = torch.autograd.grad(loss, [par[k[2:]] for k in SCALARS] + [cells])
    out = dict(image=image.detach().reshape(-1).cpu().numpy())
    out.update({k: v.cpu().numpy() for k, v in zip(SCALARS, got)})
    out.update({k: got[-1][:, q].reshape(geom.n1, geom.n2).cpu().numpy() for k, q in zip(FIELDS, (0, 1, 8))})
    return _exact_kept(out, case)


def _exact_kept(out, case):
    return out if case["form"] == "fp64" else {k: v * JANSKY if k in ("image", "spectrum") else v
                                               for k, v in out.items()}
