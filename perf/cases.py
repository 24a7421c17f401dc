"""The work that is timed: what programs built on agama_b200 have it do, through its public entry points.

A case is a dict of plain values.  `kind` says which call is made, `potential` which of the
repository's configurations it is made in, `n` how many points, particles or orbits it has:

    force      Potential.force / .eval of Cartesian points (CUDA tensors)
    hessian    Potential.forceDeriv and .density of Cartesian points (CUDA tensors)
    actions    ActionFinder(points) on CUDA tensors, or on host arrays (`host`)
    fixed      actions(potential, points, fd=one focal distance per point) on CUDA tensors
    angles     ActionFinder(points, angles=True, frequencies=True) on CUDA tensors
    orbits     orbit(potential, ic, time) for `periods` circular periods of each orbit (CUDA tensors)
    bar        orbit_target in the frame rotating with the bar: the end points and the density-grid
               row of every orbit, for `periods` to 3 x `periods` circular periods (CUDA tensors)
    finder     ActionFinder(potential): the focal-distance table and the L_circ(E) interpolator

Potentials and action finders are kept between states: a program builds them once and calls them
with many sets of points.  Everything else is made from the seed.
"""
import functools
import math

import numpy as np
import torch

import agama_b200
from agama_b200 import workloads

# the repository's benchmark potentials, and the spheroid of its fifth one without the disk, whose
# potential has the form of a one-dimensional integral (the exact values of the `fixed` cases)
POTENTIALS = {"triaxial": 1, "disk": 2, "bar": 3, "halo": 4, "galaxy": 5}
SPHEROID = dict(density=dict(type="Spheroid", mass=1, scaleRadius=1, gamma=1, beta=4, axisRatioZ=0.6),
                lmax=12, gridSizeR=80, symmetry="axisymmetric")
# inner slope and axis ratios of the density models (unit mass and scale radius)
MODELS = {"triaxial": (1.0, (1.0, 0.8, 0.6)), "bar": (0.5, (1.0, 0.7, 0.5)), "halo": (1.0, (1.0, 0.8, 0.6)),
          "galaxy": (1.0, (1.0, 1.0, 0.6)), "spheroid": (1.0, (1.0, 1.0, 0.6))}
PATTERN_SPEED = 0.05
BAR_RADIUS = 5.0                    # orbits of the bar region: starts inside five scale radii
TARGET_SHELLS, TARGET_STRIPS = 10, 2


def listed():
    return [
        # forces of a handful of test particles inside somebody's own time step: latency and launches
        {"name": "force_small", "kind": "force", "potential": "triaxial", "n": 1000},
        # forces and potentials of a snapshot
        {"name": "force_snapshot", "kind": "force", "potential": "triaxial", "n": 2000003},
        # tidal tensors and densities on a grid of points
        {"name": "hessian_grid", "kind": "hessian", "potential": "bar", "n": 400001},
        # actions of the stars of one cluster or stream
        {"name": "actions_stream", "kind": "actions", "potential": "disk", "n": 777, "host": False},
        # actions of a disk's stars, resident on the GPU: the headline workload
        {"name": "actions_disk", "kind": "actions", "potential": "disk", "n": 1000000, "host": False},
        # actions of a halo's particles from and to host arrays
        {"name": "actions_host", "kind": "actions", "potential": "halo", "n": 700001, "host": True},
        # actions with the caller's own focal distances
        {"name": "actions_fixed", "kind": "fixed", "potential": "spheroid", "n": 40001},
        # actions, angles and frequencies of a survey's stars
        {"name": "angles_survey", "kind": "angles", "potential": "galaxy", "n": 100003},
        # orbits in a triaxial galaxy: fewer than fill the GPU
        {"name": "orbits_triaxial", "kind": "orbits", "potential": "triaxial", "n": 10000, "periods": 10.0},
        # orbits in an axisymmetric galaxy: the GPU full
        {"name": "orbits_galaxy", "kind": "orbits", "potential": "galaxy", "n": 60001, "periods": 20.0},
        # an orbit library of a rotating bar with the density constraints of a Schwarzschild model
        {"name": "bar_library", "kind": "bar", "potential": "bar", "n": 3001, "periods": 10.0},
        # a new potential's action finder
        {"name": "finder", "kind": "finder", "potential": "disk", "n": 1},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["force", "hessian", "actions", "actions", "fixed", "angles", "orbits", "bar", "finder"])
    if kind == "force":
        return {"kind": kind, "potential": rng.choice(["triaxial", "bar", "disk"]), "n": size(100, 2000000)}
    if kind == "hessian":
        return {"kind": kind, "potential": rng.choice(["triaxial", "bar", "galaxy"]), "n": size(100, 400000)}
    if kind == "actions":
        return {"kind": kind, "potential": rng.choice(["disk", "halo", "galaxy"]), "n": size(50, 1000000),
                "host": rng.random() < 0.3}
    if kind == "fixed":
        return {"kind": kind, "potential": "spheroid", "n": size(50, 40000)}
    if kind == "angles":
        return {"kind": kind, "potential": rng.choice(["disk", "halo", "galaxy"]), "n": size(50, 100000)}
    if kind == "orbits":
        potential = rng.choice(["triaxial", "halo", "galaxy"])
        return {"kind": kind, "potential": potential, "n": size(50, 10000 if potential == "triaxial" else 60000),
                "periods": round(rng.uniform(2.0, 10.0 if potential == "triaxial" else 20.0), 2)}
    if kind == "bar":
        return {"kind": kind, "potential": "bar", "n": size(50, 3000), "periods": round(rng.uniform(2.0, 10.0), 2)}
    return {"kind": kind, "potential": rng.choice(["disk", "halo", "galaxy"]), "n": 1,
            "gridSizeR": rng.randrange(48, 81, 2)}


# ------------------------------------------------------------------------------------------
# what a program has in hand

@functools.lru_cache(maxsize=None)
def potential_of(name, gridSizeR=None):
    p = dict(SPHEROID if name == "spheroid" else workloads.CONFIG_POTENTIALS[POTENTIALS[name]])
    if gridSizeR:
        p["gridSizeR"] = gridSizeR
    return agama_b200.Potential(type="Multipole", **p)


@functools.lru_cache(maxsize=None)
def finder_of(name):
    return agama_b200.ActionFinder(potential_of(name))


def particles(name, n, seed):
    """phase-space points (n x 6) of the distribution that goes with the potential"""
    if name == "disk":
        return workloads.disk_particles(n, disk_vcirc, seed=seed)
    return workloads.orbit_ics(positions(name, n, seed), model_potential(name), seed=seed + 1000003)


# Speeds and times come from the density models behind the potentials and not from the engine, so
# that the inputs of a seed are the same numbers whatever evaluates the potentials.

def disk_vcirc(R):
    """circular speed of the Miyamoto-Nagai disk and NFW halo of the disk potential"""
    disk = 0.1 * R ** 2 / (R ** 2 + 3.3 ** 2) ** 1.5
    halo = np.log1p(R / 20) / R - 1 / (R + 20)
    return np.sqrt(disk + halo)


def model_potential(name):
    """positions -> potentials of the ellipsoidal model (of the bulge alone in the galaxy)"""
    gamma, axes = MODELS[name]

    def potential(x):
        x = torch.as_tensor(x)
        if torch.cuda.is_available():
            x = x.cuda()
        return torch.cat([dehnen_potential(x[k:k + 20000], gamma, axes) for k in range(0, len(x), 20000)]).cpu().numpy()
    return potential


def circular_period(gamma, E):
    """of energy E in the spherical model of the same profile (energies below the range: its inner end)"""
    r = np.logspace(-6, 8, 4001)
    mass = (r / (1 + r)) ** (3 - gamma)
    phi = -np.log1p(1 / r) if gamma == 2 else -(1 - (r / (1 + r)) ** (2 - gamma)) / (2 - gamma)
    return np.exp(np.interp(E, phi + 0.5 * mass / r, np.log(2 * np.pi * np.sqrt(r ** 3 / mass))))


def positions(name, n, seed):
    if name == "disk":
        return np.ascontiguousarray(particles(name, n, seed)[:, :3])
    gamma, axes = MODELS[name]
    return workloads.dehnen_positions(n, gamma, q=axes[1:], seed=seed)


def focal_distances(points, seed):
    """focal distances of a few tenths of the radius, as an estimate from the potential's shape gives"""
    rng = np.random.Generator(np.random.PCG64(seed + 2000003))
    return rng.uniform(0.2, 0.6, size=len(points)) * np.linalg.norm(points[:, :3], axis=1)


def bar_starts(n, seed):
    """starts inside BAR_RADIUS (a fifth of the profile's mass lies outside)"""
    pos = positions("bar", 2 * n + 100, seed)
    pos = pos[np.linalg.norm(pos, axis=1) < BAR_RADIUS][:n]
    return workloads.orbit_ics(pos, model_potential("bar"), seed=seed + 1000003)


def periods_of(name, ic):
    E = model_potential(name)(ic[:, :3]) + 0.5 * np.sum(ic[:, 3:] ** 2, axis=1)
    return circular_period(MODELS[name][0], E)


def on_gpu(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def prepare(case, seed):
    kind, name, n = case["kind"], case["potential"], case["n"]
    state = {"kind": kind}
    if kind == "finder":
        # a potential of its own for every seed: the total mass of each differs
        p = dict(workloads.CONFIG_POTENTIALS[POTENTIALS[name]])
        if case.get("gridSizeR"):
            p["gridSizeR"] = case["gridSizeR"]
        mass = 1 + 0.5 * np.random.Generator(np.random.PCG64(seed)).random()
        parts = p["density"] if isinstance(p["density"], list) else [p["density"]]
        p["density"] = [dict(d, mass=float(d["mass"] * mass)) for d in parts]
        state["potential"] = agama_b200.Potential(type="Multipole", **p)
        return state
    state["potential"] = potential_of(name)
    if kind in ("force", "hessian"):
        state["points"] = on_gpu(positions(name, n, seed))
    elif kind in ("actions", "angles"):
        w = particles(name, n, seed)
        state["finder"] = finder_of(name)
        state["points"] = w if case.get("host") else on_gpu(w)
    elif kind == "fixed":
        w = particles(name, n, seed)
        state["points"], state["fd"] = on_gpu(w), on_gpu(focal_distances(w, seed))
    elif kind == "orbits":
        ic = particles(name, n, seed)
        state["ic"], state["time"] = on_gpu(ic), on_gpu(case["periods"] * periods_of(name, ic))
    else:
        ic = bar_starts(n, seed)
        rng = np.random.Generator(np.random.PCG64(seed + 3000003))
        spread = 3.0 ** rng.uniform(size=len(ic))
        state["ic"], state["time"] = on_gpu(ic), on_gpu(case["periods"] * spread * periods_of("bar", ic))
        state["target"] = agama_b200.Target(type="DensityClassicLinear", stripsPerPane=TARGET_STRIPS,
                                            gridr=np.logspace(-1.5, 1, TARGET_SHELLS))
    return state


# ------------------------------------------------------------------------------------------
# one pass

def run(state):
    kind, pot = state["kind"], state["potential"]
    if kind == "force":
        return pot.eval(state["points"], pot=True, acc=True)
    if kind == "hessian":
        force, deriv = pot.forceDeriv(state["points"])
        return force, deriv, pot.density(state["points"])
    if kind == "actions":
        return state["finder"](state["points"])
    if kind == "fixed":
        return agama_b200.actions(pot, state["points"], fd=state["fd"])
    if kind == "angles":
        return state["finder"](state["points"], angles=True, frequencies=True)
    if kind == "orbits":
        return agama_b200.orbit(potential=pot, ic=state["ic"], time=state["time"])
    if kind == "bar":
        return agama_b200.orbit_target(pot, state["ic"], state["time"], state["target"], Omega=PATTERN_SPEED)
    return agama_b200.ActionFinder(pot).tables()


# ------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """Operations: one evaluation of a 2-D quintic cell (36 coefficients) per azimuthal harmonic with
    its gradient (150 per harmonic), and the point's coordinates, logarithm, exponential and chain
    rule (150 together); 12 evaluations and the stage sums per accepted step of an orbit, some 35
    steps per circular period; about 40 evaluations for the two integrals, the three limits and
    the constants of motion of an action, 60 with angles; about 1000 steps of the 8-dimensional shell
    problem at each of the 25 x 70 nodes of a finder."""
    kind, name, n = case["kind"], case["potential"], case["n"]
    harmonics = {"triaxial": 4, "bar": 5}.get(name, 1)
    evaluation = 150 + 150 * harmonics
    if kind == "force":
        return {"bytes": n * 8 * (3 + 4), "flops": n * evaluation}
    if kind == "hessian":
        return {"bytes": n * 8 * (3 + 3 + 6 + 1), "flops": n * (evaluation + 100 * harmonics)}
    if kind in ("actions", "fixed"):
        return {"bytes": n * 8 * (6 + 3 + (kind == "fixed")), "flops": n * 40 * evaluation}
    if kind == "angles":
        return {"bytes": n * 8 * (6 + 9), "flops": n * 60 * evaluation}
    if kind in ("orbits", "bar"):
        steps = 35 * case["periods"] * (1.8 if kind == "bar" else 1.0)
        values = 3 * TARGET_STRIPS * (TARGET_STRIPS + 1) + 1 if kind == "bar" else 0
        return {"bytes": n * (8 * (6 + 1 + 6) + 4 * TARGET_SHELLS * values),
                "flops": n * steps * 12 * (evaluation + 150)}
    return {"bytes": 8 * 25 * 70, "flops": 25 * 70 * 1000 * 12 * (evaluation + 300)}


# ------------------------------------------------------------------------------------------
# values in 64 bits, without this repository's code: the density models themselves (which the Multipole
# expansion approximates).  For a density of the ellipsoidal radius, potential and force are integrals
# over w in [0, 1] (Chandrasekhar; Binney & Tremaine, Galactic Dynamics, eq. 2.140, with
# tau = 1 / w^2 - 1); here over v = -ln w with Gauss-Legendre nodes.

def ellipsoidal_nodes(x, axes, nodes=128):
    """per point: w (n x nodes), its weights dw, and 1 - e_i w^2 for the three axes"""
    g, h = (torch.as_tensor(a, device=x.device) for a in np.polynomial.legendre.leggauss(nodes))
    top = 12 + torch.log1p(x.norm(dim=1, keepdim=True))
    w = torch.exp(-0.5 * (g + 1) * top)
    return w, 0.5 * top * h * w, [1 - (1 - a * a) * w * w for a in axes]


def dehnen_rho(m, gamma, axes):
    return (3 - gamma) / (4 * math.pi * axes[1] * axes[2]) * m ** -gamma * (1 + m) ** (gamma - 4)


def dehnen_potential(x, gamma, axes):
    w, dw, q = ellipsoidal_nodes(x, axes)
    m = w * sum(x[:, i:i + 1] ** 2 / q[i] for i in range(3)).sqrt()
    u = m / (1 + m)
    outside = (1 - u ** (2 - gamma)) / (2 - gamma) - (1 - u ** (3 - gamma)) / (3 - gamma)
    if gamma == 1:
        outside = 0.5 * (1 + m) ** -2       # the same without its cancellation at large m
    return -(3 - gamma) * (dw * outside / (q[0] * q[1] * q[2]).sqrt()).sum(1)


def dehnen_derivs(x, gamma, axes, hessian):
    """acceleration, and with hessian the derivatives of the force (xx, yy, zz, xy, yz, zx)"""
    w, dw, q = ellipsoidal_nodes(x, axes)
    m = w * sum(x[:, i:i + 1] ** 2 / q[i] for i in range(3)).sqrt()
    rho = dehnen_rho(m, gamma, axes)
    c = 4 * math.pi * axes[1] * axes[2] * dw * w * w / (q[0] * q[1] * q[2]).sqrt()
    first = [(c * rho / q[i]).sum(1) for i in range(3)]
    acc = torch.stack([-x[:, i] * first[i] for i in range(3)], 1)
    if not hessian:
        return acc, None
    slope = rho * (-gamma / m + (gamma - 4) / (1 + m)) * w * w / m      # d rho / dx_j = slope x_j / q_j
    d = []
    for i, j in ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0)):
        v = x[:, i] * x[:, j] * (c * slope / (q[i] * q[j])).sum(1)
        d.append(-(v + first[i] if i == j else v))
    return acc, torch.stack(d, 1)


def fudge_actions(w, fd, axes):
    """Staeckel-fudge actions in the axisymmetric gamma = 1 model for given focal distances (Binney
    2012): the limits by bisection, the integrals with the substitution tau = lo + (hi - lo) sin^2"""
    R = w[:, :2].norm(dim=1)
    z, D = w[:, 2], fd * fd
    vR = (w[:, 0] * w[:, 3] + w[:, 1] * w[:, 4]) / R
    vphi = (w[:, 0] * w[:, 4] - w[:, 1] * w[:, 3]) / R
    vz, L = w[:, 5], R * vphi

    def phi(lam, nu):
        r2 = ((lam - D) * (1 - nu / D)).clamp(min=0)
        return dehnen_potential(torch.stack([r2.sqrt(), 0 * r2, (lam * nu / D).clamp(min=0).sqrt()], 1), 1.0, axes)

    s = R * R + z * z
    root = ((s - D) ** 2 + 4 * R * R * D).sqrt()
    lam = 0.5 * (s + D + root)
    nu = z * z * D / lam
    p, p0 = phi(lam, nu), phi(lam, 0 * nu)
    E = p + 0.5 * (vR ** 2 + vz ** 2 + vphi ** 2)
    I3 = lam * (p - p0) + 0.5 * ((z * vphi) ** 2 + (R * vz - z * vR) ** 2 + vz ** 2 * D)
    fl = -lam * p0
    fn = fl + p * (lam - nu)

    def F_lambda(t):
        return (E * t - I3 + fn - phi(t, nu) * (t - nu)) * (t - D) - 0.5 * L * L * t

    def F_nu(t):
        return (E * t - I3 + fl - phi(lam, t) * (t - lam)) * (t - D) - 0.5 * L * L * t

    def bisect(F, inside, outside):
        for _ in range(60):
            mid = 0.5 * (inside + outside)
            ok = F(mid) > 0
            inside, outside = torch.where(ok, mid, inside), torch.where(ok, outside, mid)
        return 0.5 * (inside + outside)

    far = 2 * lam
    for _ in range(60):
        far = torch.where(F_lambda(far) > 0, 2 * far, far)
    nmax = bisect(F_nu, nu, D)
    lmin, lmax = bisect(F_lambda, lam, D), bisect(F_lambda, lam, far)
    g, h = np.polynomial.legendre.leggauss(40)
    Jr, Jz = 0 * lam, 0 * lam
    for a, b in zip(0.25 * math.pi * (g + 1), 0.25 * math.pi * h):
        jac = 2 * b * math.sin(a) * math.cos(a)
        for F, lo, hi, J in ((F_lambda, lmin, lmax, Jr), (F_nu, 0 * nmax, nmax, Jz)):
            t = lo + (hi - lo) * math.sin(a) ** 2
            J += jac * (hi - lo) * (F(t) / (2 * t)).clamp(min=0).sqrt() / (t - D).abs()
    return torch.stack([Jr / math.pi, 2 * Jz / math.pi, L], 1)


def exact(case, seed):
    kind, name, n = case["kind"], case["potential"], case["n"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind not in ("force", "hessian", "fixed") or name not in ("triaxial", "bar", "spheroid"):
        return None         # sums of models, tables and orbits have no such value
    gamma, axes = MODELS[name]
    state = prepare(case, seed)
    x = state["points"].to(device)
    parts = []
    for k in range(0, n, 20000):
        b = x[k:k + 20000]
        if kind == "fixed":
            parts.append((fudge_actions(b, state["fd"].to(device)[k:k + 20000], axes),))
        elif kind == "force":
            parts.append((dehnen_potential(b, gamma, axes), dehnen_derivs(b, gamma, axes, False)[0]))
        else:
            m = sum((b[:, i] / axes[i]) ** 2 for i in range(3)).sqrt()
            parts.append(dehnen_derivs(b, gamma, axes, True) + (dehnen_rho(m, gamma, axes),))
    out = tuple(torch.cat(p) for p in zip(*parts))
    return out[0] if kind == "fixed" else out
