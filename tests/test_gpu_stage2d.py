"""The kernel that ends a 2D stage (upwinding, divergence, viscous terms, source,
Runge-Kutta combination) at the edges of its 16 x 14 tiles, for every upwind
scheme, with and without chemistry and on both reconstructions, against the
oracle's right-hand side; and whole steps whose combination it forms against
steps completed by the kernel that sums the norm.

Tolerances: a right-hand side divides a few ulps of interface fluxes (below 3) by
the spacing (1/50 or more): 50 x 3 x 10 x 2.2e-16 = 3e-13 absolute, with a margin
of thirty for the compact systems: 1e-11.  The steps are the same operations on
the same values; only the last combination's kernel differs: 1e-14.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle
from piafs_b200 import Simulation, cases

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (16, 14), (15, 13), (17, 15), (33, 29), (47, 28)]


def flow(case, seed):
    """A smooth flow in motion with every species present, ghosted."""
    rng = np.random.default_rng(seed)
    W1, W0 = case.shape_g
    y, x = np.meshgrid((np.arange(W1) - 2.5) / (W1 - 6), (np.arange(W0) - 2.5) / (W0 - 6), indexing="ij")
    w = lambda a: a * np.sin(2 * np.pi * x + rng.uniform(0, 6)) * np.cos(2 * np.pi * y + rng.uniform(0, 6))  # noqa: E731
    rho, u, v, p = 1 + w(0.1), w(0.2), w(0.2), (1 + w(0.1)) / case.gamma
    q = [rho, rho * u, rho * v, p / (case.gamma - 1) + 0.5 * rho * (u * u + v * v)]
    if case.nvars > 4:
        q += [1 + w(0.02), 0.005 * (1 + w(0.1))] + [1e-3 * (1 + w(0.3)) for _ in range(5)]
    return np.ascontiguousarray(np.stack(q, axis=-1).reshape(-1))


def make(path, N, NY, upw, chem, scheme):
    if chem:
        cases.ns2d_photochem_beam(path, N=N, NY=NY, n_iter=4, dt=0.4 / 2048, upwinding=upw, scheme=scheme)
    else:
        cases.ns2d_shear_layer(path, N=N, NY=NY, n_iter=4, upwinding=upw, scheme=scheme)


@pytest.mark.parametrize("upw", ["llf-char", "roe", "rf-char", "rusanov"])
@pytest.mark.parametrize("chem", [False, True])
@pytest.mark.parametrize("scheme", ["weno5", "crweno5"])
def test_right_hand_side(tmp_path, upw, chem, scheme):
    for N, NY in SIZES:
        d = str(tmp_path / f"{N}x{NY}")
        make(d, N, NY, upw, chem, scheme)
        case = oracle.load(d)
        u = flow(case, N)
        t = 0.012
        want, _ = case.rhs(u, t)
        with Simulation(d) as sim:
            du = torch.from_numpy(u).cuda()
            r = torch.full_like(du, 7.0)
            sim.RHSFunction(r, du, t)
            assert np.abs(r.cpu().numpy() - want).max() <= 1e-11, (N, NY)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("chem", [False, True])
def test_steps_with_and_without_the_norm(tmp_path, chem, precision):
    d = str(tmp_path / "s")
    make(d, 33, 29, "llf-char", chem, "crweno5")
    with Simulation(d, precision) as a, Simulation(d, precision) as b:
        a.time_rk(3)
        for _ in range(3):
            b.time_rk_norm(1)
        x, y = a.state(), b.state()
        assert np.isfinite(x).all() and np.abs(x - y).max() <= 1e-14 * np.abs(y).max()
