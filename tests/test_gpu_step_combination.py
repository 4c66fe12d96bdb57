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
