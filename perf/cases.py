"""The work a user has this framework do, as cases that can be timed and compared.

Four kinds of call, each through the package's public entry points:

* ``run``   -- a simulation from an initial state: ``set_state``, ``time_rk(steps)``, ``solution``;
* ``rhs``   -- one evaluation of the right-hand side on device arrays (``RHSFunction``), as a host program that keeps
               its own time integrator calls it;
* ``host``  -- one time step on a host array in the reference layout (``time_rk_host``), the drop-in call;
* ``batch`` -- a job of many small solves on a resident ``Batch``: requests admitted, stepped together, read back and
               removed.

A case is a dict of plain values; the decks are those of ``piafs_b200.cases``.  ``exact`` is a plain torch restatement
of the same equations in 64 bits (components or characteristic WENO5, CRWENO5 with its tridiagonal systems, the four
upwind schemes, second-order viscous terms, photochemistry, SSPRK3).
"""
from __future__ import annotations

import math
import tempfile

import numpy as np
import torch

import piafs_b200
from piafs_b200 import cases as decks

G = 3                      # ghost layers
THETA = decks.THETA_RE_1E4


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one evaluation of the 1D Euler right-hand side (1024 points, WENO5, Roe)
        dict(name="rhs_1d_1024", kind="rhs", ndims=1, nx=1024, ny=1, scheme="weno5", upw="roe", weno="js",
             interp="components", chem=False, precision="fp64"),
        # the 1D density wave of the plain method, a hundred steps: launches and latency
        dict(name="run_1d_1024", kind="run", ndims=1, nx=1024, ny=1, scheme="weno5", upw="roe", weno="js",
             interp="components", chem=False, precision="fp64", steps=100),
        # a 1D line longer than one thread block serves, odd, compact scheme with the Yamaleev-Carpenter weights
        dict(name="run_1d_6001_crweno", kind="run", ndims=1, nx=6001, ny=1, scheme="crweno5", upw="llf-char",
             weno="yc", interp="components", chem=False, precision="fp64", steps=40),
        # a small photochemical grid: many short kernels a step
        dict(name="run_chem_64", kind="run", ndims=2, nx=64, ny=64, scheme="crweno5", upw="llf-char", weno="js",
             interp="components", chem=True, precision="fp64", steps=40),
        # an ordinary photochemical run, compact scheme
        dict(name="run_chem_512", kind="run", ndims=2, nx=512, ny=512, scheme="crweno5", upw="llf-char", weno="js",
             interp="components", chem=True, precision="fp64", steps=30),
        # the same physics in mixed precision, ragged sides
        dict(name="run_chem_mixed_701x500", kind="run", ndims=2, nx=701, ny=500, scheme="crweno5", upw="llf-char",
             weno="js", interp="components", chem=True, precision="mixed", steps=20),
        # explicit WENO5 with Roe upwinding on a ragged grid, one member of an ensemble run alone
        dict(name="run_chem_weno_300x217", kind="run", ndims=2, nx=300, ny=217, scheme="weno5", upw="roe", weno="js",
             interp="components", chem=True, precision="fp64", steps=40),
        # no chemistry, reconstruction on characteristic variables (the reference's default), odd sides
        dict(name="rhs_shear_char_1201x777", kind="rhs", ndims=2, nx=1201, ny=777, scheme="weno5", upw="rf-char",
             weno="js", interp="characteristic", chem=False, precision="fp64"),
        # the headline grid: one right-hand side of the 2048 x 2048 photochemical case, and one step on host arrays
        dict(name="rhs_chem_2048", kind="rhs", ndims=2, nx=2048, ny=2048, scheme="crweno5", upw="llf-char", weno="js",
             interp="components", chem=True, precision="fp64"),
        dict(name="host_chem_2048", kind="host", ndims=2, nx=2048, ny=2048, scheme="crweno5", upw="llf-char",
             weno="js", interp="components", chem=True, precision="fp64"),
        # a batched ensemble of 2D photochemical members, sides 64 .. 256 in multiples of 32
        dict(name="batch_ensemble", kind="batch", members=12, waves=0, lo=64, hi=256, mult=32, steps=30,
             precision="fp64"),
        # a serving mix in mixed precision: 1D waves and 2D beams of any side
        dict(name="batch_serving_mixed", kind="batch", members=6, waves=14, lo=64, hi=300, mult=1, steps=40,
             precision="mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["run1d", "rhs1d", "run2d", "run2d", "rhs2d", "rhs2d", "host", "batch"])
    if kind == "batch":
        mixed = rng.random() < 0.5
        return dict(kind="batch", members=rng.randint(3, 12), waves=rng.randint(0, 14) if mixed else 0, lo=64,
                    hi=_log_int(rng, 96, 256), mult=1 if mixed else 32, steps=rng.randint(10, 30),
                    precision="mixed" if mixed else "fp64")
    if kind in ("run1d", "rhs1d"):
        c = dict(kind=kind[:3], ndims=1, nx=_log_int(rng, 256, 8192), ny=1, scheme=rng.choice(["weno5", "crweno5"]),
                 upw=rng.choice(["roe", "llf-char"]), weno=rng.choice(["js", "js", "yc", "borges"]),
                 interp="components", chem=False, precision="fp64")
        if kind == "run1d":
            c["steps"] = rng.randint(20, 100)
        return c
    chem = rng.random() < 0.7
    scheme = rng.choice(["crweno5", "crweno5", "weno5"])
    c = dict(kind=kind[:3] if kind != "host" else "host", ndims=2, scheme=scheme,
             upw=rng.choice(["llf-char", "llf-char", "roe", "rf-char", "rusanov"]),
             weno=rng.choice(["js", "js", "js", "yc", "borges"]), interp="components", chem=chem, precision="fp64")
    if kind == "run2d":
        c["nx"], c["ny"] = _log_int(rng, 64, 640), _log_int(rng, 64, 640)
        c["steps"] = rng.randint(5, 30)
        if chem and scheme == "crweno5" and rng.random() < 0.4:
            c["precision"] = "mixed"
            c["upw"] = "llf-char"
    else:
        c["nx"], c["ny"] = _log_int(rng, 100, 2048), _log_int(rng, 100, 1600)
        if kind == "rhs2d" and scheme == "weno5" and rng.random() < 0.5:
            c["interp"] = "characteristic"
    return c


# ------------------------------------------------------------------ inputs
def _dt(c):
    if c["ndims"] == 1:
        return 0.1 / c["nx"]
    dt = 0.15 / max(c["nx"], c["ny"])
    return min(dt, 0.4 / 2048) if c["chem"] else dt      # the heating pulse resolved


def _deck(c, seed, path):
    weno = {"yc": {"yc": 1}, "borges": {"borges": 1}}.get(c["weno"])
    if c["ndims"] == 1:
        return decks.euler1d_density_wave(path, N=c["nx"], n_iter=10 ** 6, dt=_dt(c), amp=_amp(seed),
                                          scheme=c["scheme"], upwinding=c["upw"], weno=weno, interp=c["interp"],
                                          op_file_format="none")
    if c["chem"]:
        return decks.ns2d_photochem_beam(path, N=c["nx"], NY=c["ny"], n_iter=10 ** 6, scheme=c["scheme"],
                                         upwinding=c["upw"], seed=seed, beam_amp=5 * _amp(seed), weno=weno,
                                         interp=c["interp"], dt=_dt(c), op_file_format="none")
    return decks.ns2d_shear_layer(path, N=c["nx"], NY=c["ny"], n_iter=10 ** 6, dt=_dt(c), scheme=c["scheme"],
                                  upwinding=c["upw"], weno=weno, interp=c["interp"], amp=0.25 * _amp(seed),
                                  op_file_format="none")


def _amp(seed):
    return float(np.random.default_rng(seed).uniform(0.05, 0.3))


def _nvars(c):
    return 3 if c["ndims"] == 1 else 11 if c["chem"] else 4


def _developed(c, seed, device):
    """A flow in motion on the case's grid, [point, variable] with ghost points (zero, filled by the call): smooth
    waves of a few per cent in density, velocity, pressure and the species on the deck's background."""
    r = np.random.default_rng([seed, 17])
    nx, ny, nv = c["nx"], c["ny"], _nvars(c)
    gamma = decks.chem_gamma() if c["chem"] else 1.4
    x = (torch.arange(nx, dtype=torch.float64, device=device) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device=device) + 0.5) / ny

    def wave(a):
        s = 0.0
        for _ in range(3):
            kx, ky = int(r.integers(1, 5)), int(r.integers(1, 5))
            px, py = r.uniform(0, 2 * math.pi, 2)
            s = s + torch.cos(2 * math.pi * ky * y + py)[:, None] * torch.sin(2 * math.pi * kx * x + px)[None, :]
        return (a / 3.0) * s

    rho, p = 1.0 + wave(0.05), (1.0 + wave(0.05)) / gamma
    u, v = wave(0.1), wave(0.1)
    flow = [rho, rho * u, p / (gamma - 1.0) + 0.5 * rho * u * u] if c["ndims"] == 1 else \
        [rho, rho * u, rho * v, p / (gamma - 1.0) + 0.5 * rho * (u * u + v * v)]
    if c["chem"]:
        flow += [1.0 + wave(0.02), 0.005 * (1.0 + wave(0.1))] + [1e-3 * (1.0 + wave(0.3)) for _ in range(4)] + [wave(0.0)]
    gy = G if c["ndims"] == 2 else 0
    U = torch.zeros((ny + 2 * gy, nx + 2 * G, nv), dtype=torch.float64, device=device)
    U[gy:gy + ny, G:G + nx] = torch.stack(flow, dim=-1)
    return U


def _requests(c, seed):
    """Parameter records of a batched job: 2D beams, then 1D waves."""
    r = np.random.default_rng([seed, 29])
    out = []
    for k in range(c["members"]):
        s = math.exp(math.log(c["lo"]) + (math.log(c["hi"]) - math.log(c["lo"])) * (k + 0.5) / c["members"])
        side = max(c["mult"], int(round(s / c["mult"])) * c["mult"])
        Re = float(math.exp(r.uniform(math.log(1e3), math.log(1e5))))
        dt = min(0.4 / side, (0.4 / 2048) * 1e4 / Re, 0.1 * Re / (side * side))
        out.append(dict(kind=piafs_b200.REQUEST_NS2D_BEAM, n=side, nsteps=c["steps"], dt=dt,
                        amp=float(r.uniform(0.5, 1.5)), beam_radius=float(r.uniform(0.02, 0.1)), Re=Re, noise=1e-6,
                        seed=int(r.integers(1, 1 << 40))))
    for k in range(c["waves"]):
        n = int(round(math.exp(math.log(256) + (math.log(8192) - math.log(256)) * (k + 0.5) / c["waves"])))
        out.append(dict(kind=piafs_b200.REQUEST_EULER1D_WAVE, n=n, nsteps=c["steps"], dt=0.1 / n,
                        amp=float(r.uniform(0.05, 0.3)), beam_radius=0.0, Re=0.0, noise=0.0, seed=0))
    return out


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        return dict(c=c, batch=piafs_b200.Batch(c["precision"]),
                    reqs=[piafs_b200.Request(**q) for q in _requests(c, seed)])
    with tempfile.TemporaryDirectory() as d:
        _deck(c, seed, d)
        sim = piafs_b200.Simulation(d, c["precision"])
    s = dict(c=c, sim=sim)
    if c["kind"] == "rhs":
        s["u"] = _developed(c, seed, "cuda").reshape(-1)
        s["rhs"] = torch.empty_like(s["u"])
        s["t"] = _t_rhs()
    elif c["kind"] == "run":
        s["u0"] = sim.state()
    else:
        # a host program's state, in pinned memory; each pass advances it by one step
        buf = torch.empty(sim.shape_ghosted[0] * sim.shape_ghosted[1], dtype=torch.float64, pin_memory=True)
        s["u"], s["buf"], s["t"], s["dt"] = buf.numpy(), buf, 0.0, _dt(c)
        s["u"][:] = sim.state()
    torch.cuda.synchronize()
    return s


def _t_rhs():
    return 0.012           # inside the heating pulse


def run(state):
    s, c = state, state["c"]
    if c["kind"] == "batch":
        b = s["batch"]
        ids = [b.add_request(q) for q in s["reqs"]]
        b.step(c["steps"])
        b.poll()
        out = [b.solution(i) for i in ids]
        for i in ids:
            b.remove(i)
        return out
    sim = s["sim"]
    if c["kind"] == "rhs":
        sim.RHSFunction(s["rhs"], s["u"], s["t"])
        return {"rhs": s["rhs"], "u": s["u"]}
    if c["kind"] == "run":
        sim.set_state(s["u0"], 0.0)
        sim.time_rk(c["steps"])
        return sim.solution()
    sim.time_rk_host(s["u"], s["t"])
    s["t"] += s["dt"]
    return s["buf"]


def work(case):
    """Bytes: per RK stage the stage input and the step's state read and the stage derivative written (24 bytes a
    value), or for one right-hand side the state read and the result written; operations: reconstruction of both
    biases of u and f at every interface, upwinding, viscous terms and source."""
    c = case

    def flops(pts, nv, ndims, scheme, chem):
        recon = {"weno5": 100, "crweno5": 130}[scheme]
        return pts * (ndims * (2 * nv * recon + 200) + (150 if ndims == 2 else 0) + (80 if chem else 0))

    if c["kind"] == "batch":
        b = f = 0.0
        for q in _requests(c, 0):
            d2 = q["kind"] == piafs_b200.REQUEST_NS2D_BEAM
            pts, nv = (q["n"] ** 2, 11) if d2 else (q["n"], 3)
            b += 3 * c["steps"] * 24 * nv * pts
            f += 3 * c["steps"] * flops(pts, nv, 2 if d2 else 1, "weno5", d2)
        return {"bytes": b, "flops": f}
    pts, nv = c["nx"] * c["ny"], _nvars(c)
    one = flops(pts, nv, c["ndims"], c["scheme"], c["chem"])
    if c["kind"] == "rhs":
        return {"bytes": 16.0 * nv * pts, "flops": one}
    stages = 3 * c.get("steps", 1)
    return {"bytes": 24.0 * nv * pts * stages, "flops": one * stages}


# ------------------------------------------------------------------ the equations in 64 bits
def _phys(chem, theta):
    """gamma, Re, Pr and the viscosity and photochemistry constants of the decks (ChemistryInitialize.c defaults,
    NavierStokes2DInitialize.c)."""
    P = dict(chem=chem, gamma=1.4, Pr=0.72, Tref=273.15, T0=275.0, TS=110.4, TA=245.4, TB=27.6)
    if not chem:
        return P
    kB, NA, Ti, Ptot = 1.380649e-23, 6.02214076e23, 288.0, 101325.0
    lam, c, h, e = 2.48e-7, 3.0e8, 6.62607015e-34, 1.60217663e-19
    R = NA * kB / 0.032
    gamma = 918.45 / 650.0
    cs = math.sqrt(gamma * R * Ti)
    kg = 2 * (2 * math.pi / lam) * math.sin(theta)
    n_O2 = Ptot / (kB * Ti)
    rho_ref = Ptot / (R * Ti)
    t_ref = 1.0 / kg / cs
    P.update(gamma=gamma, Tref=Ti)
    s15 = math.exp(1.5 * math.log(Ti / P["T0"]))
    mu = 1.99e-5 * s15 * ((P["T0"] + P["TS"]) / (Ti + P["TS"]))
    kap = 2.70e-2 * s15 * ((P["T0"] + P["TA"] * math.exp(-P["TB"] / P["T0"])) /
                           (Ti + P["TA"] * math.exp(-P["TB"] / Ti)))
    P["Re"] = rho_ref * cs / kg / mu
    P["Pr"] = gamma * R / (gamma - 1) * mu / kap
    fac = kg * cs / n_O2
    k = [0.9 * 3.3e-13, 0.1 * 3.3e-13, 0.8 * 3.95e-17, 0.2 * 3.95e-17, 1.2e-16, 1.2e-16, 1.2e-17, 1.0e-17, 1.1e-16,
         2.0e-16, 0.2 * 3.0e-17]
    Ei = rho_ref * cs * cs / ((gamma - 1.0) * n_O2)
    q = [0.73, 2.8, 0.29, 0.84, 4.3, 0.81, 0.42, 1.16, 1.23, 1.81, 0.42]
    P["k"] = [v / fac for v in k]
    P["q"] = [v * e / Ei for v in q]
    P["pulse"] = 1e-8 / t_ref
    P["hnu"] = 2000.0 / 1e-8 / (c * h * (c / lam) * n_O2)
    return P


def _betas(a, b, c, d, e):
    t = 13.0 / 12.0
    return (t * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2, t * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
            t * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2)


def _weights(opt, s, kind, eps=1e-6):
    b = _betas(*s)
    if kind == "js":
        w = [o / (x + eps) ** 2 for o, x in zip(opt, b)]
    else:
        tau = (b[2] - b[0]).abs() if kind == "borges" else (s[0] - 4 * s[1] + 6 * s[2] - 4 * s[3] + s[4]) ** 2
        w = [o * (1 + (tau / (x + eps)) ** 2) for o, x in zip(opt, b)]
    t = w[0] + w[1] + w[2]
    return [x / t for x in w]


def _weno(s, kind):
    w = _weights((0.1, 0.6, 0.3), s, kind)
    a, b, c, d, e = s
    return (w[0] * (2 * a - 7 * b + 11 * c) + w[1] * (-b + 5 * c + 2 * d) + w[2] * (2 * c + 5 * d - e)) / 6


def _cells(A):
    """The cells i-3 .. i+2 of every interface i along the last dimension of a ghosted array."""
    n = A.shape[-1] - 2 * G
    return [A[..., r:r + n + 1] for r in range(6)]


def _tridiag(a, b, c, d):
    """Parallel cyclic reduction along the last dimension."""
    a, c, d = a / b, c / b, d / b
    n, k = a.shape[-1], 1
    while k < n:
        pad = lambda x, l: torch.nn.functional.pad(x, (k, 0))[..., :n] if l else torch.nn.functional.pad(x, (0, k))[..., k:]  # noqa: E731
        am, cm, dm, ap, cp, dp = pad(a, 1), pad(c, 1), pad(d, 1), pad(a, 0), pad(c, 0), pad(d, 0)
        den = 1 - a * cm - c * ap
        a, c, d = -a * am / den, -c * cp / den, (d - a * dm - c * dp) / den
        k *= 2
    return d


def _recon(A, scheme, kind):
    """(left, right) biased interface values of every line of A."""
    c = _cells(A)
    sides = []
    for s, left in ((c[:5], True), (c[:0:-1], False)):
        if scheme == "weno5":
            sides.append(_weno(s, kind))
            continue
        w = _weights((0.2, 0.5, 0.3), s, kind)
        lo, mid, hi = (2 * w[0] + w[1]) / 3, (w[0] + 2 * (w[1] + w[2])) / 3, w[2] / 3
        r = (w[0] * (s[1] + 5 * s[2]) + w[1] * (5 * s[2] + s[3]) + w[2] * (s[2] + 5 * s[3])) / 6
        ends = [_weno([x[..., :1] for x in s], kind), _weno([x[..., -1:] for x in s], kind)]
        lo, mid, hi, r = (x[..., 1:-1].clone() for x in (lo, mid, hi, r))
        a, e = (lo, hi) if left else (hi, lo)
        r[..., :1] -= a[..., :1] * ends[0]
        r[..., -1:] -= e[..., -1:] * ends[1]
        a[..., 0] = 0
        e[..., -1] = 0
        sides.append(torch.cat([ends[0], _tridiag(a, mid, e, r), ends[1]], dim=-1))
    return sides


def _prim(U, g):
    """rho, normal velocity, other velocities, pressure (the normal momentum is variable 1; the energy the last of the
    flow variables)."""
    n = 3 if U.shape[0] == 3 else 4
    rho = U[0]
    vel = [U[k] / rho for k in range(1, n - 1)]
    p = (U[n - 1] - 0.5 * rho * sum(v * v for v in vel)) * (g - 1)
    return rho, vel, p


def _flux(U, g):
    n = 3 if U.shape[0] == 3 else 4
    rho, vel, p = _prim(U, g)
    F = U * vel[0]
    F[1] += p
    F[n - 1] += p * vel[0]
    return F


def _roe(A, B, g):
    ra, va, pa = _prim(A, g)
    rb, vb, pb = _prim(B, g)
    ta, tb = ra.sqrt(), rb.sqrt()
    Ha = 0.5 * sum(v * v for v in va) + g * pa / ra / (g - 1)
    Hb = 0.5 * sum(v * v for v in vb) + g * pb / rb / (g - 1)
    vel = [(ta * x + tb * y) / (ta + tb) for x, y in zip(va, vb)]
    H = (ta * Ha + tb * Hb) / (ta + tb)
    c = ((g - 1) * (H - 0.5 * sum(v * v for v in vel))).sqrt()
    return vel, c, H


def _char(vel, c, H, g):
    """Left and right eigenvectors (fields u-c, u, [shear,] u+c) as functions on flow variables."""
    u, ek, gm = vel[0], 0.5 * sum(v * v for v in vel), g - 1

    def left(X):
        mom, E = X[1:-1], X[-1]
        dp = gm * (ek * X[0] - sum(v * m for v, m in zip(vel, mom)) + E)
        du = mom[0] - u * X[0]
        out = [(dp - c * du) / (2 * c * c), X[0] - dp / (c * c)] + [m - v * X[0] for v, m in zip(vel[1:], mom[1:])]
        return out + [(dp + c * du) / (2 * c * c)]

    def right(W):
        m, e, s, p = W[0], W[1], W[2:-1], W[-1]
        out = [m + e + p, (u - c) * m + u * e + (u + c) * p]
        out += [v * (m + e + p) + w for v, w in zip(vel[1:], s)]
        return torch.stack(out + [(H - u * c) * m + ek * e + (H + u * c) * p + sum(v * w for v, w in zip(vel[1:], s))])

    return left, right


def _speeds(A, g):
    rho, vel, p = _prim(A, g)
    return vel[0], (g * p / rho).sqrt()


def _fields(u, c, n):
    return [u - c] + [u] * (n - 2) + [u + c]


def _upwind(c, uL, uR, fL, fR, cL, cR, g):
    n = 3 if uL.shape[0] == 3 else 4
    upw = c["upw"]
    centre = n == 3 or upw in ("roe", "rusanov")
    A, B = (cL, cR) if centre else (uL, uR)
    vel, a, H = _roe(A[:n], B[:n], g)
    un, (ua, ca), (ub, cb) = vel[0], _speeds(A[:n], g), _speeds(B[:n], g)
    if upw == "rusanov":
        al = torch.maximum(torch.maximum(ca + ua.abs(), cb + ub.abs()), a + un.abs())
        return 0.5 * (fL + fR) - 0.5 * al * (uR - uL)
    left, right = _char(vel, a, H, g)
    lam = _fields(un, a, n)
    if upw == "roe":
        fix = (lambda x: torch.where(x.abs() < 1e-6, (x * x + 1e-12) / 2e-6, x.abs())) if n == 4 else torch.abs
        flow = 0.5 * (fL[:n] + fR[:n]) - right([fix(x) * w for x, w in zip(lam, left(0.5 * (uR[:n] - uL[:n])))])
        return torch.cat([flow, 0.5 * (fL[n:] + fR[n:]) - fix(un) * 0.5 * (uR[n:] - uL[n:])])

    def blend(l1, l2, l3, fl, fr, ul, ur):
        al = torch.maximum(torch.maximum(l1.abs(), l2.abs()), l3.abs())
        f = 0.5 * (fl + fr + al * (ul - ur))
        if upw == "rf-char":
            f = torch.where((l1 > 0) & (l2 > 0) & (l3 > 0), fl, torch.where((l1 < 0) & (l2 < 0) & (l3 < 0), fr, f))
        return f

    la, lb = _fields(ua, ca, n), _fields(ub, cb, n)
    w = [blend(*z) for z in zip(la, lam, lb, left(fL[:n]), left(fR[:n]), left(uL[:n]), left(uR[:n]))]
    return torch.cat([right(w), blend(ua, un, ub, fL[n:], fR[n:], uL[n:], uR[n:])])


def _hyp_dir(c, A, dxi, g):
    """dxinv (fI[i+1] - fI[i]) of lines along the last dimension; the normal momentum is variable 1."""
    F = _flux(A, g)
    cL, cR = A[..., G - 1:-G], A[..., G:-G + 1]
    if c["interp"] == "components":
        (uL, uR), (fL, fR) = _recon(A, c["scheme"], c["weno"]), _recon(F, c["scheme"], c["weno"])
    else:
        n = 3 if A.shape[0] == 3 else 4
        left, right = _char(*_roe(cL[:n], cR[:n], g), g)
        res = []
        for X in (A, F):
            W = [left(x[:n]) for x in _cells(X)]
            pair = []
            for s in (W[:5], W[:0:-1]):
                flow = right([_weno([x[k] for x in s], c["weno"]) for k in range(n)])
                pair.append(flow)
            if A.shape[0] > n:
                o = _recon(X[n:], "weno5", c["weno"])
                pair = [torch.cat([f, q]) for f, q in zip(pair, o)]
            res.append(pair)
        (uL, uR), (fL, fR) = res
    fI = _upwind(c, uL, uR, fL, fR, cL, cR, g)
    return dxi * (fI[..., 1:] - fI[..., :-1])


def _swap(U):
    """Lines along y, with the y momentum in place of the x momentum."""
    U = U.transpose(1, 2)
    return torch.cat([U[:1], U[2:3], U[1:2], U[3:]])


def _ghosts(c, U):
    nx = U.shape[2] - 2 * G
    gy = G if c["ndims"] == 2 else 0
    rows = slice(gy, U.shape[1] - gy)
    U[:, rows, :G] = U[:, rows, nx:nx + G]
    U[:, rows, nx + G:] = U[:, rows, G:2 * G]
    if gy:
        ny, g = U.shape[1] - 2 * G, 1.4          # the walls keep the gamma of physics.inp
        for k in range(G):
            for dst, src in ((k, 2 * G - 1 - k), (ny + G + k, ny + G - 1 - k)):
                rho, vel, p = _prim(U[:4, src, G:-G], g)
                U[0, dst, G:-G] = rho
                U[1, dst, G:-G] = rho * vel[0]
                U[2, dst, G:-G] = -rho * vel[1]
                U[3, dst, G:-G] = p / (g - 1) + 0.5 * rho * (vel[0] ** 2 + vel[1] ** 2)
    return U


def _dxinv(x):
    d = x[1:] - x[:-1]
    full = torch.cat([d[:1], d, d[-1:]])
    return 2.0 / (full[1:] + full[:-1])


def _viscous(U, P, dx, dy):
    g = P["gamma"]
    rho, (u, v), p = _prim(U, g)
    Q = torch.stack([u, v, g * p / rho])
    pad = lambda d: torch.cat([d[:1].expand(G), d, d[-1:].expand(G)])  # noqa: E731
    DX, DY = pad(dx)[None, None, :], pad(dy)[None, :, None]
    Qx, Qy = torch.zeros_like(Q), torch.zeros_like(Q)
    Qx[:, G:-G, :-1] = DX[..., :-1] * (Q[:, G:-G, 1:] - Q[:, G:-G, :-1])
    Qy[:, :-1, G:-G] = DY[:, :-1] * (Q[:, 1:, G:-G] - Q[:, :-1, G:-G])
    Td, T0 = Q[2] * P["Tref"], P["T0"]
    r15 = torch.exp(1.5 * torch.log(Td / T0))
    mu = r15 * (T0 + P["TS"]) / (Td + P["TS"]) / P["Re"]
    kap = r15 * (T0 + P["TA"] * math.exp(-P["TB"] / T0)) / (Td + P["TA"] * torch.exp(-P["TB"] / Td))
    kap = kap / P["Re"] / (g - 1) / P["Pr"]
    txx, tyy = 2 / 3 * mu * (2 * Qx[0] - Qy[1]), 2 / 3 * mu * (2 * Qy[1] - Qx[0])
    txy = mu * (Qy[0] + Qx[1])
    FX = torch.stack([txx, txy, u * txx + v * txy + kap * Qx[2]])
    FY = torch.stack([txy, tyy, u * txy + v * tyy + kap * Qy[2]])
    i, j = slice(G, -G), slice(G, -G)
    return dx[None, None, :] * (FX[:, j, i] - FX[:, j, G - 1:-G - 1]) + dy[None, :, None] * (FY[:, j, i] - FY[:, G - 1:-G - 1, i])


def _source(S, P, imap, t):
    k, q = P["k"], P["q"]
    f = 0.0
    if t > 0.0:
        sig = P["pulse"] / 2.35482
        f = math.exp(-(t - P["pulse"]) ** 2 / (2 * sig * sig))
    n = P["hnu"] * f * imap
    O2, O3, D1, Dg, S3, S1, CO2 = S
    src = [-(k[0] + k[1]) * n * O3 - (k[4] + k[5]) * O3 * D1 - (k[6] + k[7]) * O3 * S1 - k[9] * O3 * S3 - k[10] * Dg * O3,
           k[0] * n * O3 - (k[2] + k[3]) * D1 * O2 - (k[4] + k[5]) * D1 * O3 - k[8] * D1 * CO2,
           k[0] * n * O3 + k[9] * O3 * S3 - k[10] * Dg * O3, k[4] * O3 * D1 - k[9] * O3 * S3,
           k[2] * D1 * O2 - (k[6] + k[7]) * O3 * S1]
    Q = ((q[0] * k[0] + q[1] * k[1]) * n * O3 + (q[2] * k[2] + q[3] * k[3]) * O2 * D1 + (q[4] * k[4] + q[5] * k[5]) * O3 * D1
         + (q[6] * k[6] + q[7] * k[7]) * O3 * S1 + q[8] * k[8] * D1 * CO2 + q[9] * k[9] * O3 * S3 + q[10] * k[10] * Dg * O3)
    return src, Q / (P["gamma"] - 1)


def _rhs(c, P, U, dx, dy, imap, t):
    """Stage derivative at the interior points of a state whose ghosts are filled, [variable, row, column]."""
    g = P["gamma"]
    if c["ndims"] == 1:
        return -_hyp_dir(c, U, dx, g)
    r = -_hyp_dir(c, U[:, G:-G], dx, g) - _swap(_hyp_dir(c, _swap(U[:, :, G:-G]), dy, g))
    corner = U.clone()                      # corner ghosts are never used: any finite state there
    corner[:, :G, :G] = corner[:, :G, -G:] = corner[:, -G:, :G] = corner[:, -G:, -G:] = U[:, G:G + 1, G:G + 1]
    r[1:4] += _viscous(corner, P, dx, dy)
    if P["chem"]:
        s, q = _source(U[4:, G:-G, G:-G], P, imap, t)
        r[5:10] += torch.stack(s)
        r[3] += q
    return r


def _inner(c, U):
    return U[:, G:-G, G:-G] if c["ndims"] == 2 else U[:, :, G:-G]


def _march(c, P, U, dx, dy, imap, dt, steps):
    t = 0.0
    for _ in range(steps):
        k = []
        for cs, a in ((0.0, ()), (1.0, (1.0,)), (0.5, (0.25, 0.25))):
            V = U.clone()
            for x, d in zip(a, k):
                _inner(c, V).add_(dt * x * d)
            k.append(_rhs(c, P, _ghosts(c, V), dx, dy, imap, t + cs * dt))
        _inner(c, U).add_(dt * (k[0] / 6 + k[1] / 6 + 2 * k[2] / 3))
        t += dt
    return U


def _grid(c, device):
    ax = lambda n: (torch.arange(n, dtype=torch.float64, device=device) + (0.0 if c["ndims"] == 1 else 0.5)) / n  # noqa: E731
    return ax(c["nx"]), ax(c["ny"])


def _beam(x, y, amp, radius):
    return amp * torch.exp(-((x[None, :] - 0.5) ** 2 + (y[:, None] - 0.5) ** 2) / radius ** 2)


def _splitmix(seed, n):
    with np.errstate(over="ignore"):
        x = np.uint64(seed) * np.uint64(0x100000001B3) + np.arange(n, dtype=np.uint64) + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        x = x ^ (x >> np.uint64(31))
    return (x >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _initial(c, seed, device):
    """The initial state of a case's deck, [variable, row, column] with ghosts."""
    x, y = _grid(c, device)
    if c["ndims"] == 1:
        rho = (1.0 + _amp(seed) * torch.sin(2 * math.pi * x))[None]
        flow = [rho, rho, 1.0 / 0.4 + 0.5 * rho]
    elif c["chem"]:
        g = decks.chem_gamma()
        rho = 1.0 + np.random.default_rng(seed).uniform(-1e-6, 1e-6, size=(c["ny"], c["nx"]))
        rho = torch.from_numpy(rho).to(device)
        z = torch.zeros_like(rho)
        flow = [rho, z, z, z + 1.0 / g / (g - 1), z + 1.0, z + 0.005] + [z] * 5
    else:
        u = torch.tanh((y - 0.25) / 0.05) - torch.tanh((y - 0.75) / 0.05) - 1.0
        u, v = u[:, None] + 0.0 * x[None, :], 0.25 * _amp(seed) * torch.sin(2 * math.pi * x)[None, :] + 0.0 * y[:, None]
        flow = [torch.ones_like(u), u, v, 1.0 / 1.4 / 0.4 + 0.5 * (u * u + v * v)]
    U = torch.zeros((_nvars(c), c["ny"] + (2 * G if c["ndims"] == 2 else 0), c["nx"] + 2 * G), dtype=torch.float64, device=device)
    _inner(c, U).copy_(torch.stack(flow))
    return U


def _points(U):
    return U.permute(1, 2, 0).reshape(-1, U.shape[0]).cpu()


def exact(case, seed):
    c = case
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] == "batch":
        out = []
        for q in _requests(c, seed):
            d2 = q["kind"] == piafs_b200.REQUEST_NS2D_BEAM
            m = dict(ndims=2 if d2 else 1, nx=q["n"], ny=q["n"] if d2 else 1, scheme="weno5", weno="js", chem=d2,
                     upw="llf-char" if d2 else "roe", interp="components")
            x, y = _grid(m, device)
            U = torch.zeros((11, q["n"] + 2 * G, q["n"] + 2 * G) if d2 else (3, 1, q["n"] + 2 * G), dtype=torch.float64, device=device)
            V = _inner(m, U)
            if d2:
                P = _phys(True, math.asin(min(1.0, math.sin(THETA) * 1e4 / q["Re"])))
                noise = torch.from_numpy(_splitmix(q["seed"], q["n"] ** 2)).to(device).reshape(q["n"], q["n"])
                V[0] = 1.0 + q["noise"] * (2.0 * noise - 1.0)
                V[3] = 1.0 / P["gamma"] / (P["gamma"] - 1.0)
                V[4], V[5] = 1.0, 0.005
                imap = _beam(x, y, q["amp"], q["beam_radius"])
            else:
                P, imap = _phys(False, 0.0), None
                V[0] = 1.0 + q["amp"] * torch.sin(2 * math.pi * x)
                V[1] = V[0]
                V[2] = 1.0 / 0.4 + 0.5 * V[0]
            U = _march(m, P, U, _dxinv(x), _dxinv(y) if d2 else None, imap, q["dt"], c["steps"])
            out.append(_points(_inner(m, U)))
        return out
    P = _phys(c["chem"], THETA)
    if not c["chem"]:
        P["Re"] = 200.0
    x, y = _grid(c, device)
    dx, dy = _dxinv(x), _dxinv(y) if c["ndims"] == 2 else None
    imap = _beam(x, y, 5 * _amp(seed), 0.05) if c["chem"] else None
    if c["kind"] == "rhs":
        U = _ghosts(c, _developed(c, seed, device).permute(2, 0, 1).contiguous())
        R = torch.zeros_like(U)
        _inner(c, R).copy_(_rhs(c, P, U, dx, dy, imap, _t_rhs()))
        return {"rhs": _points(R).reshape(-1), "u": _points(U).reshape(-1)}
    U = _initial(c, seed, device)
    V = _ghosts(c, U.clone())   # the ghosts of the step's first stage, as a host array comes back with them
    U = _march(c, P, U, dx, dy, imap, _dt(c), c.get("steps", 1))
    if c["kind"] == "run":
        return _points(_inner(c, U))
    _inner(c, V).copy_(_inner(c, U))
    return _points(V).reshape(-1)
