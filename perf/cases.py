"""The calls a user of the light-curve engine makes, as timed cases.

Each case is one of
  curve    Engine.light_curve_comp, the drop-in call: one model against one
           light curve, every grid rebuilt as a fit's next step needs it
  batch    Engine.light_curve_batch_resident over models with grids of their
           own, two successive proposals of the whole ensemble per pass
  chains   sampler.ExactChi2 and the chains' curves left on the device: the
           exact half of a sampler's step, two steps per pass
  train    one training step of the surrogate network
  screen   the surrogate's two passes of a delayed-acceptance step

Parameters scatter around the detached white dwarf + M dwarf binary as a
posterior does (mass ratio, inclination, radii and temperatures a few percent
apart); points are time-ordered with jittered cadence.

Batched calls choose their flux plan by timing it, once per process and
layout, so the last bits of a batch's float64 curves change from one process
to the next; their curves and chi**2 are returned in single precision, as the
surrogate's training set keeps them.
"""
import math

import numpy as np
import torch

from lcurve_re_b200 import abi
from lcurve_re_b200 import workloads as W
from lcurve_re_b200.engine import Engine
from lcurve_re_b200.mlp import MLP
from lcurve_re_b200.model import make_data
from lcurve_re_b200.sampler import ExactChi2
from lcurve_re_b200.surrogate import NCOEF, NGRID, PARAMS, ModelFactory, Surrogate, SurrogateChi2

BINARY = dict(q=0.25, iangle=86.0, r1=0.015, r2=0.20, t1=20000.0, t2=3200.0, velocity_scale=300.0,
              ldc1_1=0.10, ldc1_2=0.60, ldc1_3=-0.45, ldc1_4=0.15,
              ldc2_1=0.70, ldc2_2=-0.60, ldc2_3=1.00, ldc2_4=-0.35,
              gravity_dark1=0.25, gravity_dark2=0.08, absorb=0.5, t0=0.0,
              beam_factor1=0.0, beam_factor2=0.0)
SIGMA = 1.5e-3
WAVELENGTH = 550.0  # nm, the models' default


def listed():
    return [
        # the smallest call: a survey light curve on coarse grids
        dict(name="curve_small", kind="curve", physics="detached", precision="mixed",
             nlat1=40, nlat2=80, npts=500, ndiv=1, diagnostics=True),
        # high-cadence photometry, finest grids, exposures split in five
        dict(name="curve_fine", kind="curve", physics="detached", precision="mixed",
             nlat1=200, nlat2=800, npts=5000, ndiv=5, diagnostics=True),
        # a likelihood call of a sampler: odd sizes, no diagnostics
        dict(name="curve_ordinary", kind="curve", physics="detached", precision="mixed",
             nlat1=81, nlat2=163, npts=2411, ndiv=1, diagnostics=False),
        # a very small white dwarf, all points around its eclipse
        dict(name="curve_tiny_star", kind="curve", physics="tiny", precision="mixed",
             nlat1=400, nlat2=200, npts=10000, ndiv=1, diagnostics=False),
        # a cataclysmic variable: opaque disc, its rim, bright spot
        dict(name="curve_disc", kind="curve", physics="disc", precision="mixed",
             nlat1=100, nlat2=200, npts=2000, ndiv=1, diagnostics=True),
        # Doppler beaming and a polynomial limb-darkening law
        dict(name="curve_beamed", kind="curve", physics="beamed", precision="mixed",
             nlat1=60, nlat2=121, npts=3001, ndiv=3, diagnostics=True),
        # the double-precision contexts, which follow the reference's sums
        dict(name="curve_fp64", kind="curve", physics="detached", precision="fp64",
             nlat1=100, nlat2=200, npts=5000, ndiv=3, diagnostics=True),
        # an ensemble of 256 models with grids from coarse to fine, all redrawn
        dict(name="batch_redrawn", kind="batch", change="all", nmodels=256, nlat2_lo=60,
             nlat2_hi=400, npts=2000),
        # the same ensemble when only the temperatures move
        dict(name="batch_temperatures", kind="batch", change="temperatures", nmodels=256,
             nlat2_lo=60, nlat2_hi=400, npts=2000),
        # the chains that passed a sampler's first stage
        dict(name="chains", kind="chains", nmodels=64, npts=1000),
        # one training step of the surrogate, forward, backward and Adam
        dict(name="train_step", kind="train", rows=4096),
        # the surrogate's part of a delayed-acceptance step
        dict(name="screen", kind="screen", rows=512, npts=1000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["curve"] * 5 + ["batch", "chains", "train", "screen"])
    if kind == "batch":
        lo = _log(rng, 40, 200)
        return dict(kind=kind, change=rng.choice(["all", "temperatures"]),
                    nmodels=_log(rng, 12, 256), nlat2_lo=lo, nlat2_hi=lo + rng.randint(0, 200),
                    npts=_log(rng, 300, 2000))
    if kind == "chains":
        return dict(kind=kind, nmodels=_log(rng, 16, 512), npts=_log(rng, 200, 2000))
    if kind == "train":
        return dict(kind=kind, rows=128 * _log(rng, 4, 64))
    if kind == "screen":
        return dict(kind=kind, rows=_log(rng, 32, 2048), npts=_log(rng, 200, NGRID))
    physics = rng.choice(["detached", "detached", "tiny", "disc", "beamed"])
    precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
    npts, ndiv = _log(rng, 200, 20000), rng.choice([1, 1, 2, 3, 5])
    nlat1, nlat2 = _log(rng, 20, 400), _log(rng, 40, 800)
    # faces x sub-exposures of the finest listed curve bound the cost; the
    # double-precision sums and the general sweeps cost several times more
    most = 2e10 if precision == "mixed" and physics in ("detached", "tiny") else 2e9
    while _faces(nlat1, nlat2) * npts * ndiv > most:
        nlat1, nlat2, npts = max(20, nlat1 * 4 // 5), max(40, nlat2 * 4 // 5), npts * 9 // 10
    return dict(kind="curve", physics=physics, precision=precision, nlat1=nlat1, nlat2=nlat2,
                npts=npts, ndiv=ndiv, diagnostics=rng.random() < 0.5)


# ---- inputs --------------------------------------------------------------------

def _parameters(rng, physics="detached"):
    p = dict(BINARY)
    p.update(q=0.25 + 0.02 * rng.standard_normal(), iangle=86.0 + 0.5 * rng.standard_normal(),
             r1=0.015 * (1 + 0.05 * rng.standard_normal()),
             r2=0.20 * (1 + 0.05 * rng.standard_normal()),
             t1=20000.0 * (1 + 0.03 * rng.standard_normal()),
             t2=3200.0 * (1 + 0.03 * rng.standard_normal()))
    if physics == "tiny":
        p.update(q=rng.uniform(0.1, 0.4), iangle=rng.uniform(85.0, 89.0), r1=rng.uniform(0.002, 0.01))
    elif physics == "beamed":
        p.update(beam_factor1=1.3, beam_factor2=1.6, ldc2_1=0.55, ldc2_2=0.15, ldc2_3=0.0, ldc2_4=0.0)
    return p


def _model(p, physics, nlat1, nlat2, rng=None):
    if physics == "disc":
        return W.cv_disc(nlat1f=nlat1, nlat2f=nlat2, nrad=60, nspot=100,
                         q=0.15 * (1 + 0.03 * rng.standard_normal()),
                         iangle=84.0 + 0.5 * rng.standard_normal(),
                         t1=p["t1"] * 0.75, temp_disc=8000.0 * (1 + 0.03 * rng.standard_normal()))
    over = dict(p, limb2="Poly") if physics == "beamed" else p
    return W.model(nlat1f=nlat1, nlat2f=nlat2, **over)


def _points(rng, physics, npts, ndiv):
    lo, hi = (-0.03, 0.03) if physics == "tiny" else (-0.2, 1.2)
    step = (hi - lo) / npts
    t = lo + step * (np.arange(npts) + rng.uniform(0.1, 0.9, npts))
    flux = 1.0 + 0.05 * np.cos(4 * np.pi * t) + SIGMA * rng.standard_normal(npts)
    return make_data(t, expose=step if ndiv > 1 else 0.0, flux=flux, ferr=SIGMA, weight=1.0,
                     ndiv=ndiv)


def _curve_inputs(case, seed):
    rng = np.random.default_rng(seed)
    p = _parameters(rng, case["physics"])
    m = _model(p, case["physics"], case["nlat1"], case["nlat2"], rng)
    return p, m, _points(rng, case["physics"], case["npts"], case["ndiv"])


def _batch_inputs(case, seed):
    """Two ensembles over the same grids: (parameters, nlat2) of each model."""
    rng = np.random.default_rng(seed)
    nlat2 = rng.integers(case["nlat2_lo"], case["nlat2_hi"] + 1, case["nmodels"])
    a = [_parameters(rng) for _ in nlat2]
    if case["change"] == "all":
        b = [_parameters(rng) for _ in nlat2]
    else:
        b = [dict(p, t1=p["t1"] * (1 + 0.01 * rng.standard_normal()),
                  t2=p["t2"] * (1 + 0.01 * rng.standard_normal())) for p in a]
    return (a, b), [int(n) for n in nlat2], _points(rng, "detached", case["npts"], 1)


def _chain_inputs(case, seed):
    rng = np.random.default_rng(seed)
    th = []
    for _ in range(2):
        rows = [_parameters(rng) for _ in range(case["nmodels"])]
        th.append(np.array([[p[k] for k in PARAMS] for p in rows]))
        th[-1][:, PARAMS.index("t0")] = 1e-3 * rng.standard_normal(case["nmodels"])
    return th, _points(rng, "detached", case["npts"], 1)


def _network_weights(seed):
    """A network as it comes from training: unit-variance activations, small
    coefficients; mean curve and smooth orthonormal components."""
    g = torch.Generator().manual_seed(seed)
    shapes = [(256, len(PARAMS))] + [(256, 256)] * 3 + [(NCOEF, 256)]
    st = {}
    for l, (o, i) in enumerate(shapes):
        st["W%d" % l] = (torch.randn(o, i, generator=g) * math.sqrt(2.0 / i)).numpy()
        st["b%d" % l] = (0.1 * torch.randn(o, generator=g)).numpy()
    t = (np.arange(NGRID) + 0.5) / NGRID
    st["basis"] = math.sqrt(2.0 / NGRID) * np.cos(np.pi * np.outer(np.arange(1, NCOEF + 1), t))
    st["mean"] = 1.0 + 0.05 * np.cos(4 * np.pi * t)
    st["cscale"] = np.array(0.02)
    return st


def _screen_inputs(case, seed):
    rng = np.random.default_rng(seed)
    index = np.sort(rng.choice(NGRID, case["npts"], replace=False))
    pts = _points(rng, "detached", case["npts"], 1)
    th = [np.array([[p[k] for k in PARAMS] for p in (_parameters(rng) for _ in range(case["rows"]))])
          for _ in range(2)]
    curves = [1.0 + 0.05 * np.cos(4 * np.pi * pts["time"]) +
              1e-3 * rng.standard_normal((case["rows"], case["npts"])) for _ in range(2)]
    return index, pts, th, curves


def prepare(case, seed):
    kind = case["kind"]
    if kind == "curve":
        _, m, d = _curve_inputs(case, seed)
        return dict(kind=kind, engine=Engine(precision=case["precision"]), model=m, data=d,
                    diagnostics=case["diagnostics"])
    if kind == "batch":
        sets, nlat2, d = _batch_inputs(case, seed)
        e = Engine()
        e.set_data(d)
        ms = [(abi.LcgModel * len(s))(*[_model(p, "detached", n // 2, n).to_c()
                                        for p, n in zip(s, nlat2)]) for s in sets]
        return dict(kind=kind, engine=e, models=ms, buffers={})
    if kind == "chains":
        th, d = _chain_inputs(case, seed)
        e = Engine()
        return dict(kind=kind, engine=e, exact=ExactChi2(e, d, ModelFactory()), theta=th,
                    curves=torch.empty(case["nmodels"], case["npts"], dtype=torch.float64,
                                       device="cuda"))
    if kind == "train":
        net = MLP(nin=len(PARAMS), nout=NCOEF, batch=case["rows"], seed=seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        net.x.copy_(torch.rand(net.B, len(PARAMS), generator=g, device="cuda") * 2 - 1)
        net.tgt.copy_(torch.randn(net.B, NCOEF, generator=g, device="cuda"))
        net.set_schedule(2e-3, 2e-5, 3000)
        return dict(kind=kind, net=net)
    index, pts, th, curves = _screen_inputs(case, seed)
    sur = Surrogate(batch=case["rows"], seed=seed)
    sur.load(_network_weights(seed))
    chi = SurrogateChi2(sur, pts, index)
    chi.bind(chi.state(th[0]), chi.anchor(curves[0]))
    chi.g_F.copy_(chi.anchor(curves[1]))
    return dict(kind=kind, chi=chi, theta=th[1])


def run(state):
    kind = state["kind"]
    if kind == "curve":
        sfac = np.ones(5)
        out = state["engine"].light_curve_comp(state["model"], state["data"], sfac=sfac,
                                               diagnostics=state["diagnostics"], no_cache=True)
        return dict(zip(("calc", "wdwarf", "chisq", "wnok", "logg1", "logg2", "rv1", "rv2"), out),
                    sfac=sfac)
    if kind == "batch":
        out = []
        for ms in state["models"]:
            calc, chisq, _, _, status = state["engine"].light_curve_batch_resident(
                ms, buffers=state["buffers"])
            out.append(dict(calc=calc.astype(np.float32), chisq=chisq.astype(np.float32),
                            status=status.copy()))
        return out
    if kind == "chains":
        out = []
        for th in state["theta"]:
            chisq = state["exact"](th)
            c = state["exact"].curves_all_device(state["curves"])
            out.append(dict(calc=c.to(torch.float32), chisq=chisq.astype(np.float32)))
        return out
    if kind == "train":
        net = state["net"]
        net.graph_step()
        nout = [w.shape[0] for w in net.W]
        return dict(dW=[g[:n] for g, n in zip(net.dW, nout)], db=net.db, W=net.W, b=net.b,
                    loss=net.loss_rows)
    chi = state["chi"]
    return dict(screen=chi.screen(state["theta"]), reverse=chi.reverse())


# ---- work ------------------------------------------------------------------------

def _faces(*nlat):
    """Faces of the latitude rings, 4 nlat**2 / pi of each grid."""
    return int(sum(4 * n * n / math.pi for n in nlat))


def work(case):
    """Flops: 16 for each face and sub-exposure where the face is turned
    towards the observer (half of them), 1000 per face whose shape and
    eclipses are solved; 2 per weight and row of the network, three times that
    with its gradients. Bytes: points in and curves out; weights, rows, curves."""
    kind = case["kind"]
    if kind == "curve":
        faces, ent = _faces(case["nlat1"], case["nlat2"]), case["npts"] * case["ndiv"]
        return dict(bytes=56 * case["npts"], flops=8 * faces * ent + 1000 * faces)
    if kind == "batch":
        faces = case["nmodels"] * _faces((case["nlat2_lo"] + case["nlat2_hi"]) / 2) * 5 // 4
        n = 2 if case["change"] == "all" else 0
        return dict(bytes=2 * (48 * case["npts"] + 8 * case["nmodels"] * case["npts"]),
                    flops=16 * faces * case["npts"] + 1000 * n * faces)
    if kind == "chains":
        faces = case["nmodels"] * _faces(40, 80)
        return dict(bytes=2 * (48 * case["npts"] + 8 * case["nmodels"] * case["npts"]),
                    flops=2 * (8 * faces * case["npts"] + 1000 * faces))
    weights = 256 * (len(PARAMS) + 3 * 256 + NCOEF)
    if kind == "train":
        # inputs and targets, and weights, moments and gradients
        return dict(bytes=4 * case["rows"] * (len(PARAMS) + NCOEF) + 4 * 7 * weights,
                    flops=6 * case["rows"] * weights)
    # two curves of each row per pass, two passes
    return dict(bytes=2 * case["rows"] * case["npts"] * 8 + 2 * weights + 4 * NCOEF * case["npts"],
                flops=2 * case["rows"] * weights + 8 * case["rows"] * case["npts"] * NCOEF)


# ---- the same quantities in 64 bits ------------------------------------------------
# Straight from the definitions, in torch's float64: the Roche surface by
# bisection, an element hidden while its line of sight dips below the
# companion's lobe potential, fluxes summed over all elements.

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _potential(q, star, x, y, z):
    """Roche potential (synchronous rotation about the star's own axis) and
    its gradient."""
    c, mu = 1 / (1 + q), q / (1 + q)
    a = (x * x + y * y + z * z) ** 0.5
    b = ((x - 1) ** 2 + y * y + z * z) ** 0.5
    ca, mb = c / a ** 3, mu / b ** 3
    xo = x if star == 0 else x - 1
    lin = mu if star == 0 else -c
    quad = (x * x + y * y) / 2 if star == 0 else 0.5 + (x * x + y * y) / 2 - x
    # star 2: centred on itself, its quadratic term carries the x of the shift
    f = -c / a - mu / b - quad + lin * x
    return f, ca * x + mb * (x - 1) - xo + lin, ca * y + mb * y - y, ca * z + mb * z


def _lobe(q):
    """Distance from star 1 to the inner Lagrangian point."""
    c, mu = 1 / (1 + q), q / (1 + q)
    lo, hi = 0.05, 0.98
    for _ in range(80):
        x = (lo + hi) / 2
        if c / x ** 2 - mu / (1 - x) ** 2 - x + mu > 0:
            lo = x
        else:
            hi = x
    return lo


def _level(q, star, r):
    """(radius of the enclosing sphere, lobe potential) of a star of radius r
    measured towards its companion."""
    lobe = _lobe(q) if star == 0 else 1 - _lobe(q)
    t = torch.tensor(r if star == 0 else 1 - r, dtype=torch.float64)
    o = torch.zeros((), dtype=torch.float64)
    return min(1.001 * r / lobe, 1.0) * lobe, float(_potential(q, star, t, o, o)[0])


def _shape(q, star, dx, dy, dz, sphere, level):
    lo, hi = torch.zeros_like(dx) + 0.02 * sphere, torch.zeros_like(dx) + sphere
    cx = 0.0 if star == 0 else 1.0
    for _ in range(60):
        r = (lo + hi) / 2
        inside = _potential(q, star, cx + r * dx, r * dy, r * dz)[0] < level
        lo, hi = torch.where(inside, r, lo), torch.where(inside, hi, r)
    return (lo + hi) / 2


def _tiles(nlat):
    th, ph, n = [], [], []
    dth = math.pi / nlat
    nl = math.ceil(math.pi / dth)
    for k in range(nl):
        t = math.pi * (k + 0.5) / nl
        m = max(16, int(2 * math.pi * math.sin(t) / dth))
        th += [t] * m
        ph += list(2 * math.pi * (np.arange(m) + 0.5) / m)
        n += [m] * m
    count = sum(max(16, int(2 * math.pi / (dth / math.sin(math.pi * (k + 0.5) / nl)))) for k in range(nl))
    return [torch.tensor(v[:count], dtype=torch.float64, device=_dev()) for v in (th, ph, n)] + [nl]


def _planck(temp):
    h, c, k = 6.6262e-34, 2.99792458e8, 1.3806e-23
    return 2e27 * h * c / (torch.exp(1e9 * h * c / k / (WAVELENGTH * temp)) - 1) / WAVELENGTH ** 3


def _elements(p, star, nlat):
    """Positions, normals, fluxes of one star's elements."""
    q, r = p["q"], p["r1"] if star == 0 else p["r2"]
    th, ph, nphi, nl = _tiles(nlat)
    d = (torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th))
    sphere, level = _level(q, star, r)
    rad = _shape(q, star, *d, sphere, level)
    cx = 0.0 if star == 0 else 1.0
    pos = (cx + rad * d[0], rad * d[1], rad * d[2])
    g = _potential(q, star, *pos)[1:]
    grav = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2) ** 0.5
    nrm = tuple(v / grav for v in g)
    one, o = torch.ones(1, dtype=torch.float64, device=th.device), torch.zeros(1, dtype=torch.float64, device=th.device)
    away = -one if star == 0 else one
    r0 = _shape(q, star, away, o, o, sphere, level)
    g0 = _potential(q, star, cx + r0 * away, o, o)[1:]
    gref = (g0[0] ** 2 + g0[1] ** 2 + g0[2] ** 2) ** 0.5
    area = (2 * math.pi / nphi * rad * torch.sin(th)) * (math.pi / nl * rad) / sum(a * b for a, b in zip(d, nrm))
    # irradiation by the other star
    v = tuple((1.0 - cx if i == 0 else 0.0) - pos[i] for i in range(3))
    dist = (v[0] ** 2 + v[1] ** 2 + v[2] ** 2) ** 0.5
    mu = sum(a * b for a, b in zip(nrm, v)) / dist
    rc = p["r2"] if star == 0 else p["r1"]
    x0 = (-mu / rc).clamp(-1, 1)
    set_ = rc * (torch.sqrt(1 - x0 * x0) * (2 + x0 * x0) / 3 - x0 * (math.pi / 2 - torch.asin(x0))) / math.pi
    geom = (rc / dist) ** 2 * torch.where(mu >= rc, mu, torch.where(mu > -rc, set_, torch.zeros_like(mu)))
    own, other = (p["t1"], p["t2"]) if star == 0 else (p["t2"], p["t1"])
    gd = p["gravity_dark1"] if star == 0 else p["gravity_dark2"]
    temp = ((own * (grav / gref) ** gd) ** 4 + p["absorb"] * other ** 4 * geom) ** 0.25
    return pos, nrm, area * _planck(temp)


def _hidden(p, star, pos):
    """Ingress and egress phase of each element behind the other star (NaN
    where it never is)."""
    other = 1 - star
    q, inc = p["q"], math.radians(p["iangle"])
    ci, si = math.cos(inc), math.sin(inc)
    sphere, level = _level(q, other, p["r2"] if other == 1 else p["r1"])
    cx = 0.0 if other == 0 else 1.0
    dx, dy, dz = pos[0] - cx, pos[1], pos[2]
    dist = (dx * dx + dy * dy) ** 0.5
    b = dz * ci - dist * si
    c = dx * dx + dy * dy + dz * dz - sphere ** 2
    cand = torch.nonzero((b < 0) & (b * b - c > 0)).flatten()
    ein, eout = torch.full_like(dx, math.nan), torch.full_like(dx, math.nan)
    if not cand.numel():
        return ein, eout
    x, y, z, dx, dy, dz, c, dist = (v[cand] for v in (*pos, dx, dy, dz, c, dist))
    half = torch.acos(((ci * dz + torch.sqrt(c.clamp(min=0))) / (si * dist)).clamp(-1, 1))
    mid = torch.atan2(dy, -dx)

    def depth(phase):
        """Least potential along the line of sight, less the lobe's."""
        ex, ey = si * torch.cos(phase), -si * torch.sin(phase)
        lam = -(ex * dx + ey * dy + ci * dz)
        reach = torch.sqrt((lam * lam - c).clamp(min=0))
        lo, hi = lam - reach, lam + reach
        for _ in range(6):  # the potential is convex near the closest approach
            _, gx, gy, gz = _potential(q, other, x + lam * ex, y + lam * ey, z + lam * ci)
            s = gx * ex + gy * ey + gz * ci
            h = 1e-5
            _, gx, gy, gz = _potential(q, other, x + (lam + h) * ex, y + (lam + h) * ey, z + (lam + h) * ci)
            cur = (gx * ex + gy * ey + gz * ci - s) / h
            lam = torch.minimum(torch.maximum(lam - s / cur.clamp(min=1e-3), lo), hi)
        return _potential(q, other, x + lam * ex, y + lam * ey, z + lam * ci)[0] - level

    lo, hi = mid - half, mid + half
    for _ in range(40):
        a, bb = lo + (hi - lo) / 3, hi - (hi - lo) / 3
        left = depth(a) < depth(bb)
        lo, hi = torch.where(left, lo, a), torch.where(left, bb, hi)
    deep = (lo + hi) / 2
    out = []
    for edge in (mid - half, mid + half):
        inn, o = deep.clone(), edge.clone()
        for _ in range(50):
            m = (inn + o) / 2
            hid = depth(m) < 0
            inn, o = torch.where(hid, m, inn), torch.where(hid, o, m)
        out.append((inn + o) / (4 * math.pi))
    hit = depth(deep) < 0
    nan = torch.full_like(x, math.nan)
    ein[cand], eout[cand] = torch.where(hit, out[0], nan), torch.where(hit, out[1], nan)
    return ein, eout


def _star_flux(p, star, elements, ranges, phases, poly):
    """Sum over the star's elements at each phase."""
    pos, nrm, flux = elements
    ein, eout = ranges
    inc = math.radians(p["iangle"])
    ld = [p["ldc%d_%d" % (star + 1, k)] for k in (1, 2, 3, 4)]
    beam = p["beam_factor%d" % (star + 1)]
    vf = p["velocity_scale"] / 2.99792458e5
    xc = p["q"] / (1 + p["q"])
    vx = -vf * pos[1]
    vy = vf * (pos[0] - xc)
    vn = nrm[0] * vx + nrm[1] * vy
    never = torch.isnan(ein)
    start = torch.where(never, torch.zeros_like(ein), ein - torch.floor(ein))
    width = torch.where(never, torch.full_like(ein, -1.0), eout - ein)
    out = torch.empty_like(phases)
    step = max(1, int(3e7 // flux.numel()))
    for k in range(0, phases.numel(), step):
        f = phases[k:k + step, None]
        ex, ey, ez = math.sin(inc) * torch.cos(2 * math.pi * f), -math.sin(inc) * torch.sin(2 * math.pi * f), math.cos(inc)
        mu = ex * nrm[0] + ey * nrm[1] + ez * nrm[2]
        if beam:
            vr = -(ex * vx + ey * vy)
            m = mu - mu * vr - vn
            v = mu * flux * (1 - beam * vr) * (m > 0)
        else:
            m, v = mu, mu * flux
        if poly:
            t = 1 - m
            v = v * (1 - t * (ld[0] + t * (ld[1] + t * (ld[2] + t * ld[3]))))
        else:
            t = torch.sqrt(m.clamp(min=0))
            v = v * (1 - sum(ld) + t * (ld[0] + t * (ld[1] + t * (ld[2] + t * ld[3]))))
        ph = f - start
        hid = (ph - torch.floor(ph)) <= width
        out[k:k + step] = torch.where((mu > 0) & ~hid, v, torch.zeros_like(v)).sum(1)
    return out


def _curve64(p, nlat1, nlat2, pts, poly=False):
    """(curve fitted to the points' scale, chi**2, star 1's flux at phase 0.5)."""
    dev = _dev()
    t = torch.tensor(pts["time"].copy(), dtype=torch.float64, device=dev) - p["t0"]
    ndiv = int(pts["ndiv"][0])
    off = [0.0] if ndiv == 1 else [(k - (ndiv - 1) / 2) / (ndiv - 1) for k in range(ndiv)]
    wgt = [1.0] if ndiv == 1 else [0.5 if k in (0, ndiv - 1) else 1.0 for k in range(ndiv)]
    phases = torch.cat([t + float(pts["expose"][0]) * o for o in off] + [torch.tensor([0.5], dtype=torch.float64, device=dev)])
    total = 0.0
    for star, nlat in ((0, nlat1), (1, nlat2)):
        el = _elements(p, star, nlat)
        f = _star_flux(p, star, el, _hidden(p, star, el[0]), phases, poly and star == 1)
        if star == 0:
            white = f[-1]
        total = total + sum(w * v for w, v in zip(wgt, f[:-1].reshape(ndiv, -1))) / max(1, ndiv - 1)
    flux, err, w = (torch.tensor(pts[k].copy(), dtype=torch.float64, device=dev) for k in ("flux", "ferr", "weight"))
    wt = w / err ** 2
    s = (wt * flux * total).sum() / (wt * total * total).sum()
    return total * s, (w * ((flux - total * s) / err) ** 2).sum(), white * s


def _net64(st, x):
    dev = _dev()
    w = {k: torch.as_tensor(v, dtype=torch.float64, device=dev) for k, v in st.items()}
    y = x
    for l in range(5):
        y = y @ w["W%d" % l].T + w["b%d" % l]
        if l < 4:
            y = torch.nn.functional.gelu(y)
    return y


def exact(case, seed):
    kind = case["kind"]
    dev = _dev()
    if kind == "curve":
        if case["physics"] == "disc":
            return None
        p, _, d = _curve_inputs(case, seed)
        calc, chisq, white = _curve64(p, case["nlat1"], case["nlat2"], d, case["physics"] == "beamed")
        return dict(calc=calc, chisq=chisq, wdwarf=white if case["diagnostics"] else None, wnok=None,
                    logg1=None, logg2=None, rv1=None, rv2=None, sfac=None)
    if kind == "batch":
        if case["nmodels"] > 20:
            return None  # a third of a second for each model and set
        sets, nlat2, d = _batch_inputs(case, seed)
        out = []
        for s in sets:
            rows = [_curve64(p, n // 2, n, d) for p, n in zip(s, nlat2)]
            out.append(dict(calc=torch.stack([r[0] for r in rows]), chisq=torch.stack([r[1] for r in rows]), status=None))
        return out
    if kind == "chains":
        if case["nmodels"] > 20:
            return None
        th, d = _chain_inputs(case, seed)
        out = []
        for t in th:
            rows = [_curve64(dict(BINARY, **dict(zip(PARAMS, r))), 40, 80, d) for r in t]
            out.append(dict(calc=torch.stack([r[0] for r in rows]), chisq=torch.stack([r[1] for r in rows])))
        return out
    if kind == "train":
        net = prepare(case, seed)["net"]  # its inputs alone
        w = [t.to(torch.float64).requires_grad_() for t in net.W]
        b = [t.to(torch.float64).requires_grad_() for t in net.b]
        y = net.x.to(torch.float64)
        for l in range(5):
            y = y @ w[l].T + b[l]
            if l < 4:
                y = torch.nn.functional.gelu(y)
        sq = ((y - net.tgt.to(torch.float64)) ** 2).sum(1)
        (sq.sum() / y.numel()).backward()
        return dict(dW=[t.grad for t in w], db=[t.grad for t in b], W=None, b=None, loss=sq.detach())
    index, pts, th, curves = _screen_inputs(case, seed)
    st = _network_weights(seed)
    lo = np.array([0.19, 84.5, 0.01275, 0.17, 18200.0, 2912.0, 0.05, 0.3, -0.005])
    hi = np.array([0.31, 87.5, 0.01725, 0.23, 21800.0, 3488.0, 0.11, 0.7, 0.005])
    coef = [_net64(st, torch.as_tensor((t - (lo + hi) / 2) / ((hi - lo) / 2), device=dev)) for t in th]
    basis = torch.as_tensor(st["basis"][:, index] * float(st["cscale"]), device=dev)
    s = [torch.as_tensor(st["mean"][index], device=dev) + c @ basis for c in coef]
    f, err = (torch.as_tensor(pts[k].copy(), device=dev) for k in ("flux", "ferr"))

    def chi2(m):
        sc = (f * m / err ** 2).sum(1) / (m * m / err ** 2).sum(1)
        return (((f - sc[:, None] * m) / err) ** 2).sum(1)
    x, y = (torch.as_tensor(c, device=dev) for c in curves)
    return dict(screen=chi2(x * s[1] / s[0]), reverse=chi2(y * s[0] / s[1]))
