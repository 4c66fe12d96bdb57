"""Whole time steps against the same steps put together here from the entry
points of their parts: the boundary fill, the hyperbolic, parabolic and source
terms of each stage, combined in torch by the tableau.  A stage's state starts
as a copy of u with its ghosts, as the reference's does, and has its ghosts
filled again.

Tolerance: a stage's terms agree to a few ulps of the interface fluxes (below 3)
over the spacing, times dt with dt over the spacing below 0.2; its combination of
at most five terms to an ulp of values below 4 a term: 3 x 10 x 2.2e-16 x 0.2 +
5 x 4 x 2.2e-16 = 6e-15 a stage.  Four stages, three steps, and a margin of ten:
1e-12.
"""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases, deck

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

Z = deck.BoundaryZone
BIG = 1e99
# stage coefficients, step coefficients, stage times
TABLEAUX = {"22": ([[], [1.0]], [0.5, 0.5], [0.0, 1.0]),
            "33": ([[], [2 / 3], [2 / 3 - 1 / 4, 1 / 4]], [1 / 4, -1 / 4, 1.0], [0.0, 2 / 3, 2 / 3]),
            "44": ([[], [0.5], [0.0, 0.5], [0.0, 0.0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6], [0.0, 0.5, 0.5, 1.0]),
            "ssprk3": ([[], [1.0], [0.25, 0.25]], [1 / 6, 1 / 6, 2 / 3], [0.0, 1.0, 0.5])}


def steps(sim, u, t, dt, rk, nsteps):
    """u (ghosted) after nsteps."""
    A, b, c = TABLEAUX[rk]
    for _ in range(nsteps):
        sim.ApplyBoundaryConditions(u)
        K = []
        for s in range(len(b)):
            Us = u.clone()
            for a, k in zip(A[s], K):
                Us += dt * a * k
            if s > 0:
                sim.ApplyBoundaryConditions(Us)
            hyp, par, src = (torch.zeros_like(u) for _ in range(3))
            sim.HyperbolicFunction(hyp, Us, t + c[s] * dt)
            sim.ParabolicFunction(par, Us, t + c[s] * dt)
            sim.SourceFunction(src, Us, t + c[s] * dt)
            K.append(par + src - hyp)
        for w, k in zip(b, K):
            u = u + dt * w * k
        t += dt
    return u


def check(d, dt, rk, u=None, nsteps=3):
    with Simulation(d) as sim:
        u = sim.state() if u is None else u
        want = steps(sim, torch.from_numpy(u.copy()).cuda(), 0.0, dt, rk, nsteps).cpu().numpy()
        sim.set_state(u, 0.0)
        sim.time_rk(nsteps)
        got = sim.state()
        assert np.isfinite(want).all() and np.abs(got - want).max() <= 1e-12


def open_faces(x="extrapolate"):
    return [Z(x, 0, 1, [0, 0, -BIG, BIG]), Z(x, 0, -1, [0, 0, -BIG, BIG]),
            Z("extrapolate", 1, 1, [-BIG, BIG, 0, 0]), Z("extrapolate", 1, -1, [-BIG, BIG, 0, 0])]


def walls():
    return open_faces("periodic")[:2] + [Z("slip-wall", 1, f, [-BIG, BIG, 0, 0], [0.0, 0.0]) for f in (1, -1)]


@pytest.mark.parametrize("zones,N,NY", [(open_faces(), 40, 2), (open_faces(), 2, 40), (open_faces(), 40, 1),
                                        (open_faces(), 2, 2), (open_faces(), 40, 3), (walls(), 40, 2),
                                        (walls(), 40, 1)])
@pytest.mark.parametrize("rk", ["33", "44", "ssprk3"])
def test_grids_narrower_than_their_ghosts(tmp_path, rk, zones, N, NY):
    """There the boundary fill of one face reads ghosts of the face across,
    which a stage's state has from u."""
    d = str(tmp_path / "n")
    cases.ns2d_channel(d, zones, N=N, NY=NY, n_iter=3, dt=2e-3, par="2", time_scheme_type=rk, flow=(0.3, 0.2),
                       bump=0.2, bump_at=(0.4, 0.3), bump_radius=0.4)
    check(d, 2e-3, rk)


LINE_ENDS = {"periodic": None,
             "walls": [Z("slip-wall", 0, 1, [0.0, 0.0], [0.1]), Z("slip-wall", 0, -1, [0.0, 0.0], [0.0])],
             "fixed": [Z("dirichlet", 0, 1, [0.0, 0.0], values=[1.0, 1.0, 3.0]), Z("extrapolate", 0, -1, [0.0, 0.0])]}


@pytest.mark.parametrize("scheme,upw,weno,N,rk,ends", [
    ("weno5", "roe", None, 16, "33", "periodic"), ("weno5", "roe", None, 129, "44", "walls"),
    ("weno5", "llf-char", {"yc": 1}, 257, "ssprk3", "fixed"), ("weno5", "rf-char", {"mapped": 1}, 1009, "22", "walls"),
    ("weno5", "rusanov", {"borges": 1}, 8192, "ssprk3", "periodic"), ("upw5", "roe", None, 300, "44", "fixed"),
    ("crweno5", "roe", None, 17, "44", "walls"), ("crweno5", "llf-char", {"yc": 1}, 259, "33", "fixed"),
    ("crweno5", "rusanov", None, 700, "ssprk3", "walls"), ("crweno5", "rf-char", {"mapped": 1}, 4097, "22", "periodic"),
    ("crweno5", "roe", {"borges": 1}, 6001, "ssprk3", "fixed")])
def test_lines(tmp_path, scheme, upw, weno, N, rk, ends):
    """1D lines whose whole steps are one launch."""
    d = str(tmp_path / "l")
    cases.euler1d_density_wave(d, N=N, n_iter=3, dt=0.1 / N, scheme=scheme, upwinding=upw, weno=weno,
                               time_scheme_type=rk, zones=LINE_ENDS[ends])
    check(d, 0.1 / N, rk)


@pytest.mark.parametrize("scheme,N", [("weno5", n) for n in (8, 17, 63, 64, 127, 128, 255, 1024, 2047, 4099, 10240, 10241)]
                         + [("crweno5", n) for n in (16, 255, 256, 257, 258, 513, 1024, 4096, 4098, 4100, 8193, 8194)])
def test_line_sizes(tmp_path, scheme, N):
    """Where segments and clusters begin and end (8, 258, 8194 and 10241 points:
    lines of separate kernels)."""
    d = str(tmp_path / "l")
    cases.euler1d_density_wave(d, N=N, n_iter=3, dt=0.1 / N, scheme=scheme)
    check(d, 0.1 / N, "ssprk3")


@pytest.mark.parametrize("scheme", ["weno5", "crweno5"])
@pytest.mark.parametrize("ends", ["periodic", "walls", "fixed"])
@pytest.mark.parametrize("rk", ["22", "33", "44", "ssprk3"])
def test_line_ends(tmp_path, scheme, ends, rk):
    d = str(tmp_path / "l")
    cases.euler1d_density_wave(d, N=150, n_iter=3, dt=0.1 / 150, scheme=scheme, time_scheme_type=rk,
                               weno={"no_limiting": 1} if ends == "periodic" else None, zones=LINE_ENDS[ends])
    check(d, 0.1 / 150, rk)


@pytest.mark.parametrize("rk", ["22", "33", "44", "ssprk3"])
@pytest.mark.parametrize("layers", [0, 1, 2])
@pytest.mark.parametrize("N,NY,scheme,upw", [(33, 29, "crweno5", "llf-char"), (200, 230, "weno5", "roe")])
def test_grids(tmp_path, N, NY, scheme, upw, layers, rk):
    """The combination formed by the kernel that ends a stage, on either side of
    148 tiles of 16 x 14, for 4, 11 and 18 variables: what a wall leaves of the
    passive variables' ghosts, corners included, is u's in every stage.  There
    every ghost gets a value of its own."""
    d = str(tmp_path / "g")
    cases.ns2d_photochem_beam(d, N=N, NY=NY, n_iter=3, dt=2e-4, scheme=scheme, upwinding=upw, time_scheme_type=rk,
                              chemistry=layers > 0, layers=max(layers, 1), noise=1e-2, flow=(0.2, 0.1), zones=walls(),
                              extra_chem={"z_mm": 1.3} if layers == 2 else None)
    with Simulation(d) as sim:
        u = sim.state().reshape(NY + 6, N + 6, -1)
        sim.ApplyBoundaryConditions(t := torch.from_numpy(u).cuda().contiguous())
        u = t.cpu().numpy()
    rng = np.random.default_rng(N)
    for a, b in ((slice(0, 3), slice(None)), (slice(NY + 3, None), slice(None)), (slice(None), slice(0, 3)),
                 (slice(None), slice(N + 3, None))):
        u[a, b] = 1.0 + 0.1 * rng.uniform(size=u[a, b].shape)
    check(d, 2e-4, rk, u.reshape(-1))
