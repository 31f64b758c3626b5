"""Performance cases: the work that users of this framework have it do, through its public entry points.

Families:

* ``eval``      potential, gradient or Hessian at n points (``AbstractPotential`` methods);
* ``orbit``     ``evaluate_orbit`` of n orbits on one save grid (adaptive or constant step, saves or dense output);
* ``uneven``    ``dynamics.integrate`` of a batch with its own span and save grid per orbit;
* ``subhalos``  the plain direct sum: Milky Way plus many Plummer subhalos, constant step;
* ``adjoint``   gradients of a terminal loss through constant-step orbits (``adjoint.orbit_adjoint``);
* ``stream``    gradient of a track loss through a stream with a moving progenitor (``stream.gradient``);
* ``mock``      ``MockStreamGenerator.run`` from host arrays to host arrays;
* ``train``     training of the potential surrogate (``surrogate.train``);
* ``surrogate`` orbits under the learned surrogate (``surrogate.integrate``).

A case is a dict of plain values; ``listed`` gives the fixed ones, ``draw`` one more of the same ranges.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import galax_gb300 as gx
from galax_gb300 import adjoint, dynamics, stream, surrogate
from galax_gb300.potential import CompositePotential, PlummerPotential

G = 4.498502151469553e-12  # kpc^3 / (Msun Myr^2)
KMS = 0.001022712165045695  # kpc/Myr per km/s
F64 = torch.float64
# MilkyWayPotential's parameters: disk (m, a, b), halo (m, r_s), bulge and nucleus (m, r_s)
DISK, HALO, BULGE, NUCLEUS = (6.8e10, 3.0, 0.28), (5.4e11, 15.62), (5e9, 1.0), (1.71e9, 0.07)
# counted floating-point operations per accepted step in MilkyWayPotential, and per gradient, by method
STEP_FLOPS, GRAD_FLOPS = {5: 1002.0, 8: 2276.0}, 80.0
STAGES = {5: 6, 8: 13}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a handful of points, as an interactive user or a host-side optimiser asks for them: latency
        {"name": "gradient_1k", "family": "eval", "what": "gradient", "pot": "mw", "n": 1000},
        # a map of tidal fields over a particle snapshot
        {"name": "hessian_4m", "family": "eval", "what": "hessian", "pot": "mw", "n": 4_194_304},
        # the commonest call of all: one orbit with the default integrator
        {"name": "orbit_1", "family": "orbit", "pot": "mw", "n": 1, "method": 8, "dt": 0.0, "T": 2000.0,
         "saves": 256, "dense": False},
        # the small plain workload of the benchmark: 1,024 orbits, Dopri8 dt = 1 Myr, 1 Gyr, 100 saves
        {"name": "orbits_plain_1024", "family": "orbit", "pot": "mw", "n": 1024, "method": 8, "dt": 1.0, "T": 1000.0,
         "saves": 100, "dense": False},
        # a cluster's or survey's stars in a composite that is a component table, default integrator, odd sizes
        {"name": "orbits_mw2022_3001", "family": "orbit", "pot": "mw2022", "n": 3001, "method": 8, "dt": 0.0,
         "T": 1500.0, "saves": 77, "dense": False},
        # the benchmark's uneven batch (a quarter of its orbits): spans 0.1-5 Gyr, 10-1000 saves each
        {"name": "uneven_65536", "family": "uneven", "n": 65_536, "T": 5000.0, "saves": 1000},
        # the plain path that the surrogate stands in for, at a batch of a few thousand orbits
        {"name": "subhalos_16384", "family": "subhalos", "n": 16_384, "k": 512, "steps": 100},
        # the differentiation workload (a quarter of its orbits, an eighth of its span)
        {"name": "adjoint_16384", "family": "adjoint", "n": 16_384, "method": 8, "dt": 0.5, "steps": 500, "ckpt": 256},
        # the stream-gradient workload (a sixth of its releases)
        {"name": "stream_grad_500", "family": "stream", "releases": 500, "df": "offsets", "ckpt": 0},
        # a mock stream as galax's users make one: host arrays in, two arms out
        {"name": "mock_stream_1000", "family": "mock", "releases": 1000, "T": 3000.0},
        # a few epochs of surrogate training (the full run is 400 epochs on 4M points)
        {"name": "train_262144", "family": "train", "n": 262_144, "epochs": 4, "batch": 8192},
        # orbits under the surrogate with its exact near field: an eighth of the benchmark's, 20 steps
        {"name": "surrogate_131072", "family": "surrogate", "n": 131_072, "steps": 20, "near": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["eval", "eval", "orbit", "orbit", "orbit", "uneven", "subhalos", "adjoint", "stream", "mock",
                         "train", "surrogate"])
    if family == "eval":
        pot = rng.choice(["mw", "mw", "mw_sub"])
        return {"family": family, "what": rng.choice(["potential", "gradient", "hessian"]), "pot": pot,
                "n": _log_int(rng, 1, 4_194_304 if pot == "mw" else 262_144)}
    if family == "orbit":
        dt = rng.choice([0.0, 0.0, 1.0])
        dense = rng.random() < 0.2
        return {"family": family, "pot": rng.choice(["mw", "mw", "mw2022", "bovy", "mw_linear"]),
                "n": _log_int(rng, 1, 512 if dense else 4096), "method": rng.choice([5, 8, 8]), "dt": dt,
                "T": float(_log_int(rng, 100, 1000 if dt else 2000)), "saves": _log_int(rng, 2, 300), "dense": dense}
    if family == "uneven":
        return {"family": family, "n": _log_int(rng, 300, 65_536), "T": float(_log_int(rng, 500, 5000)),
                "saves": _log_int(rng, 20, 1000)}
    if family == "subhalos":
        return {"family": family, "n": _log_int(rng, 64, 16_384), "k": _log_int(rng, 32, 512),
                "steps": _log_int(rng, 20, 100)}
    if family == "adjoint":
        return {"family": family, "n": _log_int(rng, 64, 16_384), "method": rng.choice([5, 8, 8]), "dt": 0.5,
                "steps": _log_int(rng, 50, 500), "ckpt": rng.choice([16, 100, 256])}
    if family == "stream":
        return {"family": family, "releases": _log_int(rng, 50, 500),
                "df": rng.choice(["offsets", "fardal2015", "chen2024"]), "ckpt": rng.choice([0, 0, 64])}
    if family == "mock":
        return {"family": family, "releases": _log_int(rng, 50, 1000), "T": float(_log_int(rng, 500, 3000))}
    if family == "train":
        return {"family": family, "n": _log_int(rng, 20_000, 262_144), "epochs": rng.choice([1, 2, 4]),
                "batch": rng.choice([8192, 4096, 5000])}
    return {"family": family, "n": _log_int(rng, 500, 131_072), "steps": _log_int(rng, 5, 20),
            "near": rng.random() < 0.7}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, lo, hi):
    return torch.rand(n, generator=g, device="cuda", dtype=F64) * (hi - lo) + lo


def _isotropic(g, n):
    v = torch.randn((n, 3), generator=g, device="cuda", dtype=F64)
    return v / v.norm(dim=1, keepdim=True)


def _mw_gradient(x):
    """grad Phi of MilkyWayPotential at x (n, 3)."""
    r = x.norm(dim=1)
    f = G * HALO[0] * (torch.log1p(r / HALO[1]) / r**3 - 1 / (r**2 * (HALO[1] + r)))
    for m, c in (BULGE, NUCLEUS):
        f = f + G * m / (r * (r + c) ** 2)
    m, a, b = DISK
    zb = torch.sqrt(x[:, 2] ** 2 + b * b)
    u = G * m / (x[:, 0] ** 2 + x[:, 1] ** 2 + (zb + a) ** 2) ** 1.5
    return torch.stack([(u + f) * x[:, 0], (u + f) * x[:, 1], (u * (zb + a) / zb + f) * x[:, 2]], dim=1)


def _circular_speed(x):
    return torch.sqrt((x * _mw_gradient(x)).sum(1).abs())


def _disk_like(g, n):
    """(n, 6): radii U(4, 20) kpc, isotropic directions, azimuthal circular speed times N(1, 0.1), N(0, 20 km/s) in z."""
    x = _isotropic(g, n) * _uniform(g, n, 4.0, 20.0)[:, None]
    vc, R = _circular_speed(x), torch.hypot(x[:, 0], x[:, 1])
    phi = torch.stack([-x[:, 1] / R, x[:, 0] / R, torch.zeros_like(R)], dim=1)
    noise = torch.randn((n, 4), generator=g, device="cuda", dtype=F64)
    v = vc[:, None] * phi * (1.0 + 0.1 * noise[:, :3])
    v[:, 2] += 20.0 * KMS * noise[:, 3]
    return torch.cat([x, v], dim=1)


def _plunging(g, n):
    """(n, 6): radii log-uniform 0.5-100 kpc, circular speed times U(0.3, 1.1) in random tangential directions."""
    rhat = _isotropic(g, n)
    x = rhat * torch.exp(_uniform(g, n, math.log(0.5), math.log(100.0)))[:, None]
    a = _isotropic(g, n)
    a = a - (a * rhat).sum(1, keepdim=True) * rhat
    a = a / a.norm(dim=1, keepdim=True)
    return torch.cat([x, a * (_circular_speed(x) * _uniform(g, n, 0.3, 1.1))[:, None]], dim=1)


def _subhalos(seed, k):
    """Masses, scale radii and centres of k Plummer subhalos."""
    rng = np.random.default_rng(seed)
    m = np.exp(rng.uniform(np.log(1e6), np.log(1e8), k))
    b = rng.uniform(0.1, 1.0, k)
    d = rng.normal(size=(k, 3))
    return m, b, d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(5.0, 50.0, k)[:, None]


def _plummers(seed, k):
    m, b, c = _subhalos(seed, k)
    return CompositePotential([PlummerPotential(m_tot=m[i], r_s=b[i], origin=tuple(c[i])) for i in range(k)])


def _potential(kind, seed=0):
    if kind == "mw2022":
        return gx.MilkyWayPotential2022()
    if kind == "bovy":
        return gx.BovyMWPotential2014()
    if kind == "mw_linear":  # a halo that grows by a third over 3 Gyr
        return gx.MilkyWayPotential(halo={"m": gx.LinearParameter(slope=6e7, point_time=0.0, point_value=HALO[0])})
    if kind == "mw_sub":
        return CompositePotential([gx.MilkyWayPotential(), _plummers(seed, 64)])
    return gx.MilkyWayPotential()


def _points(g, n):
    return _isotropic(g, n) * torch.exp(_uniform(g, n, math.log(0.1), math.log(200.0)))[:, None]


def _integrator(method, dt, **pid):
    solver = gx.Dopri8() if method == 8 else gx.Dopri5()
    if dt:
        return gx.Integrator(solver=solver, stepsize_controller=gx.ConstantStepSize(), dt0=dt)
    return gx.Integrator(solver=solver, stepsize_controller=gx.PIDController(**(pid or {"rtol": 1e-7, "atol": 1e-7})))


def _prepare_uneven(case, g):
    n = case["n"]
    y0 = _plunging(g, n)
    dur = torch.exp(_uniform(g, n, math.log(100.0), math.log(case["T"])))
    # the same grid sizes for every seed, so that the outputs of all seeds have one shape
    ns = torch.randint(10, case["saves"] + 1, (n,), generator=_gen(11), device="cuda")
    offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    offs[1:] = torch.cumsum(ns, 0)
    orbit = torch.repeat_interleave(torch.arange(n, device="cuda"), ns)
    k = torch.arange(int(offs[-1]), device="cuda") - offs[orbit]
    ts = dur[orbit] * (k / (ns[orbit] - 1))
    ts[offs[1:] - 1] = dur
    return {"pot": gx.MilkyWayPotential(), "y0": y0, "t1": dur, "ts": ts, "offs": offs,
            "cfg": _integrator(5, 0.0, rtol=1e-8, atol=1e-10).config()}


def prepare(case, seed):
    family, g = case["family"], _gen(seed)
    s = {"family": family}
    if family == "eval":
        s.update(pot=_potential(case["pot"], seed), x=_points(g, case["n"]), what=case["what"])
    elif family == "orbit":
        s.update(pot=_potential(case["pot"]), w0=_disk_like(g, case["n"]), dense=case["dense"],
                 t=torch.linspace(0.0, case["T"], case["saves"], dtype=F64, device="cuda"),
                 integrator=_integrator(case["method"], case["dt"]))
    elif family == "uneven":
        s.update(_prepare_uneven(case, g))
    elif family == "subhalos":
        s.update(pot=CompositePotential([gx.MilkyWayPotential(), _plummers(seed, case["k"])]),
                 y0=_disk_like(g, case["n"]), T=float(case["steps"]), cfg=_integrator(5, 1.0).config())
        s["ts"] = torch.tensor([s["T"]], dtype=F64, device="cuda")
    elif family == "adjoint":
        y0, t1 = _disk_like(g, case["n"]), case["steps"] * case["dt"]
        pert = torch.randn(y0.shape, generator=g, device="cuda", dtype=F64)
        pert *= torch.tensor([0.1] * 3 + [2.0 * KMS] * 3, dtype=F64, device="cuda")
        cfg = _integrator(case["method"], case["dt"]).config()
        pot = gx.MilkyWayPotential()
        end, _, _ = dynamics.integrate(pot, y0, 0.0, t1, torch.tensor([t1], dtype=F64, device="cuda"), cfg)
        s.update(pot=pot, y0=y0, t1=t1, dt=case["dt"], target=end[:, 0, :].t() + pert, method=case["method"],
                 ckpt=case["ckpt"])
    elif family == "stream":
        n = case["releases"]
        pot = gx.MilkyWayPotential()
        vc = float(_circular_speed(torch.tensor([[20.0, 0.0, 0.0]], dtype=F64, device="cuda"))[0])
        speed, inc = 0.6 * vc * (1.0 + 0.02 * math.sin(seed)), math.radians(30.0)
        w_now = [20.0, 0.0, 0.0, 0.0, speed * math.cos(inc), speed * math.sin(inc)]
        cfg = stream.config(n_release=n, dt=1.0, w_now=w_now, prog_m=1e5, prog_b=0.02, method=8, k_ckpt=case["ckpt"],
                            df=case["df"])
        columns = {"offsets": 12, "fardal2015": 4, "chen2024": 6}[case["df"]]
        noise = torch.randn((n, columns), generator=g, device="cuda", dtype=F64)
        pert = torch.randn((2 * n, 6), generator=g, device="cuda", dtype=F64)
        pert *= torch.tensor([0.1] * 3 + [2.0 * KMS] * 3, dtype=F64, device="cuda")
        s.update(pot=pot, cfg=cfg, noise=noise, target=stream.simulate(pot, cfg, noise).final + pert)
    elif family == "mock":
        rng = np.random.default_rng(seed)
        n = case["releases"]
        w0 = np.array([14.0, 2.0, 6.0, -0.02, 0.15, 0.06]) * rng.uniform(0.95, 1.05, 6)
        s.update(gen=gx.MockStreamGenerator(gx.FardalStreamDF(), gx.MilkyWayPotential()), w0=w0,
                 ts=np.linspace(0.0, case["T"], n), draws=rng.normal(size=(n, 4)))
    elif family == "train":
        x = _points(g, case["n"])
        sub = _plummers(seed, 64)
        s.update(x=x, phi=sub.potential(x), grad=sub.gradient(x), epochs=case["epochs"], batch=case["batch"])
    else:
        # a network of the trained one's size whose term has the subhalos' share of the potential
        mlp = surrogate.MLPSurrogate(surrogate.init_params(seed), 50.0, 2e-4)
        near = surrogate.ShortRange(_plummers(seed, 512), 12.0) if case["near"] else None
        s.update(pot=gx.MilkyWayPotential(), mlp=mlp, near=near, y0=_disk_like(g, case["n"]), t1=float(case["steps"]))
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    family = s["family"]
    if family == "eval":
        return getattr(s["pot"], s["what"])(s["x"])
    if family == "orbit":
        o = gx.evaluate_orbit(s["pot"], s["w0"], s["t"], integrator=s["integrator"], dense=s["dense"])
        return [o.q, o.p] if s["dense"] else [o.q, o.p, o.status, o.steps]
    if family == "uneven":
        return dynamics.integrate(s["pot"], s["y0"], 0.0, s["t1"], s["ts"], s["cfg"], save_offsets=s["offs"])
    if family == "subhalos":
        return dynamics.integrate(s["pot"], s["y0"], 0.0, s["T"], s["ts"], s["cfg"])
    if family == "adjoint":
        r = adjoint.orbit_adjoint(s["pot"], s["y0"], 0.0, s["t1"], dt=s["dt"], target=s["target"],
                                  method=s["method"], k_ckpt=s["ckpt"])
        return [r.yT, r.grad_y0, r.grad_params]
    if family == "stream":
        r = stream.gradient(s["pot"], s["cfg"], s["noise"], s["target"])
        return [r.final, r.grad_params, r.grad_w_now, r.loss]
    if family == "mock":
        arms, last = s["gen"].run(None, s["ts"], s["w0"], 1e5, draws=s["draws"])
        return [arms["lead"].q, arms["lead"].p, arms["trail"].q, arms["trail"].p, last]
    if family == "train":
        mlp, report = surrogate.train(s["x"], s["phi"], s["grad"], length_scale=50.0, epochs=s["epochs"],
                                      batch=s["batch"])
        return [mlp.params, report.loss]
    return surrogate.integrate(s["pot"], s["mlp"], s["y0"], 0.0, s["t1"], 1.0, near=s["near"])


def work(case):
    """Inputs and outputs once each; operations of the steps that the orbits take (adaptive ones: as many as they
    take on average over these inputs)."""
    family = case["family"]
    if family == "eval":
        out = {"potential": 1, "gradient": 3, "hessian": 9}[case["what"]]
        per = {"potential": 50, "gradient": 80, "hessian": 160}[case["what"]]
        return {"bytes": 8.0 * case["n"] * (3 + out), "flops": case["n"] * (per + (64 * 20 if case["pot"] == "mw_sub" else 0))}
    if family == "orbit":
        per_gyr = {5: 260.0, 8: 110.0}[case["method"]]  # default tolerances
        steps = case["T"] / case["dt"] if case["dt"] else 4 + per_gyr * case["T"] / 1000.0
        if case["method"] == 8:  # a save inside a step is one more partial step
            steps += case["saves"]
        return {"bytes": 8.0 * case["n"] * 6 * (1 + case["saves"]), "flops": case["n"] * steps * STEP_FLOPS[case["method"]]}
    if family == "uneven":
        span = (case["T"] - 100.0) / math.log(case["T"] / 100.0)
        saves = 0.5 * (10 + case["saves"])
        return {"bytes": 8.0 * case["n"] * (6 + 2 + 7 * saves), "flops": case["n"] * 1.25 * span * STEP_FLOPS[5]}
    if family == "subhalos":
        return {"bytes": 8.0 * case["n"] * 12, "flops": case["n"] * case["steps"] * (STEP_FLOPS[5] + 6.0 * 20 * case["k"])}
    if family == "adjoint":  # forward, recomputation and a reverse sweep of about twice the forward step
        return {"bytes": 8.0 * case["n"] * 24, "flops": 4.0 * case["n"] * case["steps"] * STEP_FLOPS[case["method"]]}
    if family == "stream":
        n = case["releases"]
        steps = n * (n + 1) + 2 * n  # two particles per release, and the progenitor there and back
        return {"bytes": 8.0 * n * (12 + 36), "flops": 4.0 * steps * STEP_FLOPS[8]}
    if family == "mock":
        steps = case["releases"] * (110.0 * case["T"] / 1000.0 + 4)  # two particles, half the span on average
        return {"bytes": 8.0 * case["releases"] * 24, "flops": steps * STEP_FLOPS[8]}
    if family == "train":
        per = 2.0 * (12 * 256 * 256 + 6 * 256 * 256)  # twelve layer products and six weight-gradient terms
        batch = min(case["batch"], case["n"])
        points = float(case["n"] // batch * batch * case["epochs"])
        return {"bytes": points * 28.0, "flops": points * per}
    per = 6 * (2.0 * (6 * 256 * 256 + 3 * 256 * 2)) + STEP_FLOPS[5]
    return {"bytes": 8.0 * case["n"] * 12, "flops": case["n"] * case["steps"] * per}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _sphere_terms(kind, r):
    """g(r) with grad Phi = g x, and g'(r)/r, of the centred spheres of MilkyWayPotential."""
    if kind == "halo":
        m, c = HALO
        L, q = torch.log1p(r / c), c + r
        return G * m * (L / r**3 - 1 / (r * r * q)), G * m * (3 / (r**4 * q) - 3 * L / r**5 + 1 / (r**3 * q * q))
    m, c = BULGE if kind == "bulge" else NUCLEUS
    q = r + c
    return G * m / (r * q * q), -G * m * (3 * r + c) / (r**3 * q**3)


def _exact_eval(what, x, plummers):
    n = x.shape[0]
    r = x.norm(dim=1)
    m, a, b = DISK
    zb = torch.sqrt(x[:, 2] ** 2 + b * b)
    D = torch.sqrt(x[:, 0] ** 2 + x[:, 1] ** 2 + (zb + a) ** 2)
    if what == "potential":
        out = -G * m / D - G * HALO[0] * torch.log1p(r / HALO[1]) / r
        for mass, c in (BULGE, NUCLEUS):
            out = out - G * mass / (r + c)
    elif what == "gradient":
        out = _mw_gradient(x)
    else:
        v = torch.stack([x[:, 0], x[:, 1], x[:, 2] * (zb + a) / zb], dim=1)
        u, w = G * m / D**3, 3 * G * m / D**5
        diag = torch.stack([u, u, u * (1 + a * b * b / zb**3)], dim=1)
        out = torch.diag_embed(diag) - w[:, None, None] * v[:, :, None] * v[:, None, :]
        eye = torch.eye(3, dtype=F64, device="cuda")
        for kind in ("halo", "bulge", "nucleus"):
            g, gpr = _sphere_terms(kind, r)
            out = out + g[:, None, None] * eye + gpr[:, None, None] * x[:, :, None] * x[:, None, :]
    for mass, c, origin in plummers:
        d = x - origin
        s2 = (d * d).sum(1) + c * c
        if what == "potential":
            out = out - G * mass / torch.sqrt(s2)
        elif what == "gradient":
            out = out + (G * mass / s2**1.5)[:, None] * d
        else:
            g = G * mass / s2**1.5
            out = out + g[:, None, None] * torch.eye(3, dtype=F64, device="cuda")
            out = out - (3 * g / s2)[:, None, None] * d[:, :, None] * d[:, None, :]
    return out.reshape(n, *out.shape[1:])


def _plummer_list(seed, k):
    m, b, c = _subhalos(seed, k)
    return [(m[i], b[i], torch.as_tensor(c[i], dtype=F64, device="cuda")) for i in range(k)]


# the Runge-Kutta pairs' rows: Dormand & Prince (1980) and Prince & Dormand (1981)
_A5 = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
       [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
       [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656]]
_B5 = [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]
_A8 = [[], [1 / 18], [1 / 48, 1 / 16], [1 / 32, 0, 3 / 32], [5 / 16, 0, -75 / 64, 75 / 64],
       [3 / 80, 0, 0, 3 / 16, 3 / 20],
       [29443841 / 614563906, 0, 0, 77736538 / 692538347, -28693883 / 1125000000, 23124283 / 1800000000],
       [16016141 / 946692911, 0, 0, 61564180 / 158732637, 22789713 / 633445777, 545815736 / 2771057229,
        -180193667 / 1043307555],
       [39632708 / 573591083, 0, 0, -433636366 / 683701615, -421739975 / 2616292301, 100302831 / 723423059,
        790204164 / 839813087, 800635310 / 3783071287],
       [246121993 / 1340847787, 0, 0, -37695042795 / 15268766246, -309121744 / 1061227803, -12992083 / 490766935,
        6005943493 / 2108947869, 393006217 / 1396673457, 123872331 / 1001029789],
       [-1028468189 / 846180014, 0, 0, 8478235783 / 508512852, 1311729495 / 1432422823, -10304129995 / 1701304382,
        -48777925059 / 3047939560, 15336726248 / 1032824649, -45442868181 / 3398467696, 3065993473 / 597172653],
       [185892177 / 718116043, 0, 0, -3185094517 / 667107341, -477755414 / 1098053517, -703635378 / 230739211,
        5731566787 / 1027545527, 5232866602 / 850066563, -4093664535 / 808688257, 3962137247 / 1805957418,
        65686358 / 487910083],
       [403863854 / 491063109, 0, 0, -5068492393 / 434740067, -411421997 / 543043805, 652783627 / 914296604,
        11173962825 / 925320556, -13158990841 / 6184727034, 3936647629 / 1978049680, -160528059 / 685178525,
        248638103 / 1413531060, 0]]
_B8 = [14005451 / 335480064, 0, 0, 0, 0, -59238493 / 1068277825, 181606767 / 758867731, 561292985 / 797845732,
       -1041891430 / 1371343529, 760417239 / 1151165299, 118820643 / 751138087, -528747749 / 2220607170, 1 / 4]


def _rk_step(gradient, y, h, method):
    rows, last = (_A8, _B8) if method == 8 else (_A5, _B5)
    slopes = []
    for row in rows + [last]:
        z = y
        for a, f in zip(row, slopes):
            if a:
                z = z + (h * a) * f
        if len(slopes) == len(rows):
            return z
        slopes.append(torch.cat([z[:, 3:], -gradient(z[:, :3])], dim=1))


def exact(case, seed):
    family = case["family"]
    if family == "eval":
        x = _points(_gen(seed), case["n"])
        return _exact_eval(case["what"], x, _plummer_list(seed, 64) if case["pot"] == "mw_sub" else [])
    if family == "orbit" and case["dt"] and case["method"] == 8 and case["pot"] == "mw" and not case["dense"]:
        y, dt = _disk_like(_gen(seed), case["n"]), case["dt"]
        t = torch.linspace(0.0, case["T"], case["saves"], dtype=F64, device="cuda").tolist()
        saves, k = [], 0
        for ts in t:
            while (k + 1) * dt <= ts:
                y, k = _rk_step(_mw_gradient, y, dt, 8), k + 1
            saves.append(_rk_step(_mw_gradient, y, ts - k * dt, 8) if ts > k * dt else y)
        w = torch.stack(saves, dim=1)
        return [w[..., :3], w[..., 3:], None, None]
    if family == "subhalos":
        y, plummers = _disk_like(_gen(seed), case["n"]), _subhalos(seed, case["k"])
        m, b, c = (torch.as_tensor(v, dtype=F64, device="cuda") for v in plummers)

        def gradient(x):
            d = x[:, None, :] - c
            f = G * m / ((d * d).sum(2) + b * b) ** 1.5
            return _mw_gradient(x) + (f[:, :, None] * d).sum(1)

        for _ in range(case["steps"]):
            y = _rk_step(gradient, y, 1.0, 5)
        return [y.t()[:, None, :], None, None]
    if family == "adjoint":
        y = _disk_like(_gen(seed), case["n"])
        for _ in range(case["steps"]):
            y = _rk_step(_mw_gradient, y, case["dt"], case["method"])
        return [y, None, None]
    return None
