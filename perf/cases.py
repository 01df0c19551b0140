"""The work a user has this framework do, as timed cases.

Two programs call it.  One is a deck run: some KDK steps, then a frame
(positions and velocities as FP32 rows) and the conservation diagnostics, as
the deck front end does for every frame it writes (kinds ``deck``, ``adaptive``,
``block``).  The other is a host integrator that replaces its force function:
it hands new positions over and takes the accelerations back (kind ``accel``).

Every system turns slowly, moves and sits off the origin (a cluster on its
orbit), so its centre of mass, momentum and angular momentum are figures of
their own and not the rounding left of a zero.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("opengl-physics_gb300")

OFFSET = (0.3, -0.2, 0.1)   # bulk position and velocity of every system
BULK = (0.2, 0.1, -0.15)
ENERGY_MAX_N = 262144       # largest system whose pair potential the diagnostics sum by default
EXACT_MAX_PAIRS = 2e11      # pair terms a 64-bit direct reference may take


def _case(name, kind, n, model="plummer", **kw):
    c = dict(name=name, kind=kind, n=n, model=model, leaf=16, eps=0.01, theta=0.5, dt=1e-3, steps=4,
             precision="split", softening="plummer", mac="geometric", nsys=1)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a host integrator's force function on a thousand bodies
        _case("accel_1k", "accel", 1000, "ball", leaf=8, eps=0.05),
        # the reference's own demonstration deck: 2,048 bodies, frames of 5 steps
        _case("deck_2k", "deck", 2048, eps=0.05, steps=5),
        # block timesteps (rungs up to 8), the size the block-step tests use
        _case("block_4k", "block", 4096, leaf=8, dt=0.01, steps=1),
        # the reference's CPU benchmark: 16,384 bodies, 10 steps
        _case("deck_16k", "deck", 16384, steps=10),
        # spline softening under the adaptive step rule, an odd size
        _case("adaptive_20k", "adaptive", 20011, leaf=8, softening="spline", eps=0.05),
        # the force function with the relative (per-particle) opening test
        _case("accel_rel_50k", "accel", 49999, leaf=8, mac="relative"),
        # a mid-size deck; the frame's energy is the exact pair sum
        _case("deck_131k", "deck", 131071),
        # one million bodies in plain FP32
        _case("plain_1m", "deck", 1048576, eps=0.005, dt=5e-4, precision="plain"),
        # independent systems of uneven size advanced together
        _case("ensemble_64", "deck", 0, nsys=64, theta=0.6, leaf=32, steps=2),
        # the galaxy at 4,194,304 bodies with the geometric opening test
        _case("theta_4m", "deck", 4194304, "galaxy", leaf=40, eps=0.002, theta=0.63, dt=2e-4),
        # the same galaxy with the learned opening test and its periodic check
        _case("learned_4m", "deck", 4194304, "galaxy", leaf=48, eps=0.002, theta=0.63, dt=2e-4, steps=10,
              mac="learned", budget=3.3e-4),
        # the largest: cold collapse of 16,777,216 bodies, learned test
        _case("collapse_16m", "deck", 16777216, "ball", leaf=32, eps=0.001, theta=0.6, dt=1e-4, mac="learned",
              budget=1.7e-4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("accel", "accel", "deck", "deck", "deck", "large", "large", "adaptive", "block", "ensemble"))
    opt = dict(leaf=rng.choice((8, 12, 16, 24, 32, 40, 48, 64)), theta=round(rng.uniform(0.45, 0.8), 3),
               eps=round(math.exp(rng.uniform(math.log(0.002), math.log(0.05))), 5), steps=rng.randint(2, 6))
    prec = rng.choice(("split", "split", "plain"))
    soft = rng.choice(("plummer", "plummer", "spline"))
    if kind == "accel":
        return _drawn(_case("", "accel", _log(rng, 500, 200000), rng.choice(("plummer", "ball", "galaxy")),
                            precision=prec, softening=soft, mac=rng.choice(("geometric", "relative")), **opt))
    if kind == "deck":
        n = _log(rng, 1000, 65536 if soft == "spline" else 131072)
        return _drawn(_case("", "deck", n, rng.choice(("plummer", "galaxy")), precision=prec, softening=soft, **opt))
    if kind == "large":
        learned = rng.random() < 0.5
        if learned:
            opt.update(budget=round(rng.uniform(2e-4, 6e-4), 6), leaf=rng.choice((32, 40, 48, 64)))
        opt.update(eps=0.002, theta=max(opt["theta"], 0.55), steps=min(opt["steps"], 4))
        return _drawn(_case("", "deck", _log(rng, ENERGY_MAX_N + 1, 4194304), "galaxy" if learned else
                            rng.choice(("plummer", "galaxy")), precision="split" if learned else prec, dt=2e-4,
                            mac="learned" if learned else "geometric", **opt))
    if kind == "adaptive":
        return _drawn(_case("", "adaptive", _log(rng, 1000, 40000), precision=prec, softening=soft, **opt))
    if kind == "block":
        opt.update(steps=1, eps=max(opt["eps"], 0.01))
        return _drawn(_case("", "block", _log(rng, 1000, 16384), precision=prec, dt=0.01, **opt))
    opt["steps"] = rng.randint(1, 3)
    return _drawn(_case("", "deck", rng.randint(0, 1 << 20), nsys=rng.randint(3, 64), **opt))


def _drawn(c):
    del c["name"]
    return c


# ---- inputs -----------------------------------------------------------------

def _directions(g, n):
    u = torch.randn(3, n, generator=g, device="cuda", dtype=torch.float64)
    return u / u.norm(dim=0)


def _rand(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64).clamp_(1e-12, 1 - 1e-12)


def _plummer(g, n):
    """Plummer sphere, r < 20a, velocities of its distribution function."""
    r = (_rand(g, n) * (20.0 ** 3 / 401.0 ** 1.5)).pow(-2.0 / 3.0).sub(1.0).rsqrt()
    q = torch.linspace(0, 1, 4097, device="cuda", dtype=torch.float64)
    cdf = torch.cumsum(q * q * (1 - q * q).clamp_min(0).pow(3.5), 0)
    cdf = cdf / cdf[-1]
    u = _rand(g, n)
    k = torch.searchsorted(cdf, u).clamp_(1, 4096)
    speed = q[k - 1] + (q[k] - q[k - 1]) * (u - cdf[k - 1]) / (cdf[k] - cdf[k - 1])
    v = speed * math.sqrt(2.0) * (1 + r * r).pow(-0.25)
    return _directions(g, n) * r, _directions(g, n) * v, torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)


def _galaxy(g, n):
    """Hernquist halo (mass 0.9, isotropic Jeans dispersion) and exponential
    disk (mass 0.1, circular speed plus 10 % dispersion)."""
    nd = n // 10
    nh = n - nd
    s = _rand(g, nh).sqrt() * (30.0 / 31.0)
    r = s / (1 - s)
    t = 12 * r * (1 + r) ** 3 * torch.log1p(1 / r) - r / (1 + r) * (25 + 52 * r + 42 * r * r + 12 * r ** 3)
    x = _directions(g, nh) * r
    v = torch.randn(3, nh, generator=g, device="cuda", dtype=torch.float64) * (0.075 * t).clamp_min(0).sqrt()
    R = (-0.2 * (_rand(g, nd) * _rand(g, nd)).log()) % 2.0
    phi = 2 * math.pi * _rand(g, nd)
    z = 0.02 * torch.atanh(2 * _rand(g, nd) - 1)
    inner = 0.1 * (1 - (1 + R / 0.2) * torch.exp(-R / 0.2)) + 0.9 * R * R / (R + 1) ** 2
    vc = (inner / R.clamp_min(1e-9)).sqrt()
    dv = torch.randn(3, nd, generator=g, device="cuda", dtype=torch.float64) * 0.1 * vc
    xd = torch.stack([R * phi.cos(), R * phi.sin(), z])
    vd = torch.stack([-vc * phi.sin(), vc * phi.cos(), torch.zeros_like(vc)]) + dv
    m = torch.cat([torch.full((k,), w / max(k, 1), device="cuda", dtype=torch.float64) for k, w in ((nh, 0.9), (nd, 0.1))])
    return torch.cat([x, xd], 1), torch.cat([v, vd], 1), m


def _ball(g, n):
    """Uniform ball, cold."""
    x = _directions(g, n) * _rand(g, n).pow(1.0 / 3.0)
    return x, torch.zeros_like(x), torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)


MODELS = {"plummer": _plummer, "galaxy": _galaxy, "ball": _ball}


def _sizes(case):
    """Particles per system: log-uniform in [1,024, 65,536] for an ensemble,
    whose ``n`` seeds them (the same systems for every seed of the inputs)."""
    if case["nsys"] == 1:
        return [case["n"]]
    u = np.random.RandomState(case["n"]).uniform(math.log(1024), math.log(65536), case["nsys"])
    return [int(round(math.exp(v))) for v in u]


def _inputs(case, seed):
    """(positions, velocities, masses) on the GPU as FP32 values in FP64."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    parts = [MODELS[case["model"]](g, n) for n in _sizes(case)]
    x, v, m = (torch.cat([p[k] for p in parts], -1) for k in range(3))
    v += 0.3 * torch.stack([-x[1], x[0], torch.zeros_like(x[2])]) / (1 + (x * x).sum(0))
    x += torch.tensor(OFFSET, device="cuda", dtype=torch.float64)[:, None]
    v += torch.tensor(BULK, device="cuda", dtype=torch.float64)[:, None]
    return x.float().double(), v.float().double(), m.float().double()


def _system(case, x, v, m):
    sim = pkg.NBodySystem(pkg.StepParams(G=1.0, eps=case["eps"], theta=case["theta"], dt=case["dt"]),
                          leaf_capacity=case["leaf"],
                          precision=pkg.PRECISION_SPLIT if case["precision"] == "split" else pkg.PRECISION_PLAIN,
                          mac=pkg.MAC_RELATIVE if case["mac"] == "relative" else pkg.MAC_GEOMETRIC)
    if case["softening"] == "spline":
        sim.set_softening(pkg.SOFTENING_SPLINE)
    sim.set_particles_f32(*(a.float().cpu().numpy() for a in (*x, *v, m)))
    if case["nsys"] > 1:
        sim.set_ensemble(np.concatenate([[0], np.cumsum(_sizes(case))]))
    return sim


def prepare(case, seed):
    x, v, m = _inputs(case, seed)
    sim = _system(case, x, v, m)
    if case["mac"] == "learned":
        sim.lmac_train(snapshots=1, steps_between=0, dt=0.0, pairs=1 << 18, epochs=6, batch=2048, seed=1)
        # the check runs once in every pass; its threshold leaves the learned test on
        sim.lmac_set_opts(budget=case["budget"], check_every=case["steps"], check_targets=1024, revert_rms=0.02,
                          screen=300.0 if case["model"] == "ball" else 1000.0)
        sim.set_opts(mac=pkg.MAC_LEARNED)
    sim.prime()
    state = {"case": case, "sim": sim}
    if case["kind"] == "accel":  # the host integrator's own arrays, a little further on
        state["host"] = [a.cpu().numpy() for a in x + case["dt"] * v]
    return state


# ---- one pass ---------------------------------------------------------------

def run(state):
    case, sim = state["case"], state["sim"]
    if case["kind"] == "accel":
        sim.set_state(*state["host"])
        # the accelerations are FP32 values that the call widens; kept as the
        # FP32 rows a frame has
        return {"acc": np.stack(sim.compute_accel(), axis=1, dtype=np.float32, casting="same_kind")}
    if case["kind"] == "deck":
        sim.step(case["steps"], case["dt"])
    elif case["kind"] == "adaptive":
        for _ in range(case["steps"]):
            sim.step(1, sim.adaptive_dt(0.025, case["dt"]))
    else:
        for _ in range(case["steps"]):
            sim.block_step(case["dt"], eta=0.025, max_rung=8)
    pos, vel = sim.frame_f32()
    diags = [sim.diagnostics()] if case["nsys"] == 1 else sim.ensemble_diagnostics()
    return {"pos": pos, "vel": vel, **{k: np.array([d[k] for d in diags])
                                       for k in ("kinetic", "potential", "com", "L", "P")}}


# ---- what a pass cannot do without ------------------------------------------

def _terms(theta, n):
    """Interactions per particle of a tree walk at this opening angle: the
    classical 28 pi / 9 theta^-3 log_8 count of a uniform system."""
    return min(n, 28 * math.pi / 9 / theta ** 3 * max(1.0, math.log(max(n * theta ** 3, 8.0), 8)))


def work(case):
    sizes = _sizes(case)
    n = sum(sizes)
    # at equal error the learned test opens about as much as theta 1 would
    theta = 1.0 if case["mac"] == "learned" else case["theta"]
    evals = 1 if case["kind"] == "accel" else case["steps"] * (4 if case["kind"] == "block" else 1)
    flops = 60.0 * evals * sum(k * _terms(theta, k) for k in sizes)
    state = 80 if case["precision"] == "split" else 48  # position, velocity and acceleration of a particle
    if case["kind"] == "accel":
        return {"bytes": n * (24 + 24 + state), "flops": flops}
    pairs = n * (n - 1) / 2 if n <= ENERGY_MAX_N else 0
    return {"bytes": n * (2 * state * evals + 24 + state), "flops": flops + 10.0 * pairs}


# ---- the same in 64 bits, by direct summation -------------------------------

def _chi(q):
    """Enclosed-mass fraction of the cubic spline kernel at q = r / h."""
    t = (2 - q).clamp_min(0)
    a = q ** 3 * (4 / 3 - 1.2 * q ** 2 + 0.5 * q ** 3)
    b = 1 - 4 * (t ** 4 / 4 - t ** 5 / 5 + t ** 6 / 24)
    return torch.where(q < 1, a, b)


def _phi(q):
    """Pair potential of the spline kernel, in units of G m m / h."""
    t = (2 - q).clamp_min(0)
    a = -(1.4 - 2 / 3 * q ** 2 + 0.3 * q ** 4 - 0.1 * q ** 5)
    b = -((1 - 4 * (t ** 4 / 4 - t ** 5 / 5 + t ** 6 / 24)) / q.clamp_min(1e-300) + t ** 4 / 2 - t ** 5 / 5)
    return torch.where(q < 1, a, b)


def _pairs(case, x, m, energy=False):
    """Direct accelerations (3, n), or the pair potential when ``energy``."""
    spline, eps = case["softening"] == "spline", case["eps"]
    n = x.shape[1]
    out, pot = torch.empty_like(x), 0.0
    step = max(1, (1 << 25) // n)
    for i in range(0, n, step):
        j = min(n, i + step)
        d = [x[k][None, :] - x[k][i:j, None] for k in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        if spline:
            r = r2.sqrt()
            w = _phi(r / eps) / eps if energy else torch.where(r2 > 0, _chi(r / eps) / (r2 * r), 0.0)
        else:
            ir = r2.add_(eps * eps).rsqrt_()
            w = -ir if energy else ir * ir * ir
        if energy:
            w[torch.arange(j - i), torch.arange(i, j)] = 0.0
            pot += 0.5 * float(m[i:j] @ (w @ m))
        else:
            w *= m[None, :]
            for k in range(3):
                out[k, i:j] = torch.einsum("ij,ij->i", w, d[k])
    return pot if energy else out


def _forces(case, x, m):
    parts, at = [], 0
    for n in _sizes(case):
        parts.append(_pairs(case, x[:, at:at + n], m[at:at + n]))
        at += n
    return torch.cat(parts, 1)


def _block_step(case, x, v, a, m):
    dt, eta, top = case["dt"], 0.025, 8
    tau = eta * (case["eps"] / a.norm(dim=0)).sqrt()
    rung = torch.where(tau < dt, torch.ceil(torch.log2(dt / tau)).clamp_max(top), torch.zeros_like(tau)).long()
    rmax = int(rung.max())
    units = 2 ** (rmax - rung)
    half = 0.5 * dt / 2.0 ** rung
    for sub in range(2 ** rmax):
        v = v + torch.where(sub % units == 0, half, torch.zeros_like(half)) * a
        x = x + dt / 2 ** rmax * v
        ends = (sub + 1) % units == 0
        a = torch.where(ends, _forces(case, x, m), a)
        v = v + torch.where(ends, half, torch.zeros_like(half)) * a
    return x, v, a


def exact(case, seed):
    sizes = _sizes(case)
    evals = {"accel": 1, "block": 256 * case["steps"]}.get(case["kind"], case["steps"] + 1)
    if sum(n * n for n in sizes) * evals > EXACT_MAX_PAIRS:
        return None
    x, v, m = _inputs(case, seed)
    if case["kind"] == "accel":
        return {"acc": _forces(case, x + case["dt"] * v, m).T.contiguous()}
    a = _forces(case, x, m)
    for _ in range(case["steps"]):
        if case["kind"] == "block":
            x, v, a = _block_step(case, x, v, a, m)
            continue
        dt = case["dt"]
        if case["kind"] == "adaptive":
            dt = min(max(0.025 * math.sqrt(case["eps"] / float(a.norm(dim=0).max())), dt / 4096), dt)
        v = v + 0.5 * dt * a
        x = x + dt * v
        a = _forces(case, x, m)
        v = v + 0.5 * dt * a
    out = {"pos": x.T.contiguous(), "vel": v.T.contiguous(), "kinetic": [], "com": [], "L": [], "P": []}
    at = 0
    for n in sizes:
        xs, vs, ms = x[:, at:at + n], v[:, at:at + n], m[at:at + n]
        at += n
        com = (ms * xs).sum(1) / ms.sum()
        out["kinetic"].append(0.5 * (ms * vs * vs).sum())
        out["com"].append(com)
        out["L"].append((ms * torch.linalg.cross(xs - com[:, None], vs, dim=0)).sum(1))
        out["P"].append((ms * vs).sum(1))
    out.update({k: torch.stack(w) for k, w in out.items() if isinstance(w, list)})
    # the diagnostics sum the potential up to ENERGY_MAX_N bodies, of one system only
    out["potential"] = np.array([_pairs(case, x, m, energy=True)]) if len(sizes) == 1 and sizes[0] <= ENERGY_MAX_N else None
    return out
