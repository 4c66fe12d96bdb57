"""1D Euler steps in one launch (a cluster of CTAs holding the line) against
the kernel-by-kernel steps of the same deck, which a step with the residual
norm takes: the whole ghosted state and the clock after five steps, at the
sizes where segments and clusters begin and end and over the boundary types,
tableaux, weights and upwind schemes the path accepts.

Tolerance: the same formulas per point and stage; the compiler may fuse
multiply-adds differently, a few ulps of the state per stage.  Fifteen stages
of at most 4 ulps (2.2e-16 each), values of at most 5, with a margin of ten:
1e-12.
"""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases, deck

pytestmark = pytest.mark.gpu
Z = deck.BoundaryZone
WALLS = [Z("slip-wall", 0, 1, [0.0, 0.0], [0.1]), Z("slip-wall", 0, -1, [0.0, 0.0], [0.0])]
OPEN = [Z("extrapolate", 0, 1, [0.0, 0.0]), Z("reflect", 0, -1, [0.0, 0.0])]
FIXED = [Z("dirichlet", 0, 1, [0.0, 0.0], values=[1.0, 1.0, 3.0]), Z("extrapolate", 0, -1, [0.0, 0.0])]


def both(tmp_path, N, nsteps=5, **kw):
    d = str(tmp_path / f"n{N}")
    cases.euler1d_density_wave(d, N=N, n_iter=nsteps, dt=0.1 / N, **kw)
    with Simulation(d) as a, Simulation(d) as b:
        a.time_rk(nsteps)
        for _ in range(nsteps):
            b.time_rk_norm(1)
        assert a.info["t"] == b.info["t"] and a.info["iter"] == b.info["iter"]
        return a.state(), b.state()


def check(got, want):
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    f = np.isfinite(want)      # a reflected density is negative: NaN spreads from that end, alike on both paths
    assert np.abs(got[f] - want[f]).max(initial=0.0) <= 1e-12


@pytest.mark.parametrize("N", [8, 16, 17, 63, 64, 127, 128, 129, 255, 257, 1009, 1024, 2047, 4099, 8192, 10240, 10241])
def test_sizes(tmp_path, N):
    check(*both(tmp_path, N))


@pytest.mark.parametrize("scheme,upwinding,weno", [
    ("weno5", "llf-char", None), ("weno5", "rf-char", {"mapped": 1}), ("weno5", "rusanov", {"borges": 1}),
    ("weno5", "roe", {"yc": 1}), ("weno5", "roe", {"no_limiting": 1}), ("upw5", "roe", None)])
def test_schemes(tmp_path, scheme, upwinding, weno):
    check(*both(tmp_path, 301, scheme=scheme, upwinding=upwinding, weno=weno))


@pytest.mark.parametrize("zones", [WALLS, OPEN, FIXED], ids=["walls", "open", "fixed"])
@pytest.mark.parametrize("rk", ["1fe", "22", "33", "44", "ssprk3"])
def test_boundaries_and_tableaux(tmp_path, zones, rk):
    check(*both(tmp_path, 150, zones=zones, time_scheme_type=rk))


# CRWENO5: a warp a system up to 4097 points in CTAs of 256 rows, two beyond in
# CTAs of 512 (258: two cells in the last CTA, kernel by kernel)
@pytest.mark.parametrize("N", [16, 17, 255, 256, 257, 258, 259, 513, 1024, 4096, 4097, 4098, 4100, 6001, 8193, 8194])
def test_compact_sizes(tmp_path, N):
    check(*both(tmp_path, N, scheme="crweno5"))


@pytest.mark.parametrize("upwinding,weno", [("llf-char", {"yc": 1}), ("rf-char", {"mapped": 1}),
                                            ("rusanov", {"borges": 1}), ("roe", {"no_limiting": 1})])
@pytest.mark.parametrize("zones", [None, WALLS, OPEN, FIXED], ids=["periodic", "walls", "open", "fixed"])
def test_compact_schemes(tmp_path, upwinding, weno, zones):
    check(*both(tmp_path, 700, scheme="crweno5", upwinding=upwinding, weno=weno, zones=zones))


@pytest.mark.parametrize("scheme", ["weno5", "crweno5"])
@pytest.mark.parametrize("zones", [None, WALLS, OPEN, FIXED], ids=["periodic", "walls", "open", "fixed"])
@pytest.mark.parametrize("N", [65, 600])
def test_right_hand_side(tmp_path, scheme, zones, N):
    """RHSFunction in one launch against minus the divergence of
    HyperbolicFunction on the state with its ghosts filled: interior, zero
    ghosts, and the ghosts it fills in u.  A right-hand side divides interface
    rounding (a few ulps of values below 10) by the spacing."""
    torch = pytest.importorskip("torch")
    d = str(tmp_path / "r")
    cases.euler1d_density_wave(d, N=N, n_iter=1, dt=0.1 / N, scheme=scheme, zones=zones)
    with Simulation(d) as sim:
        u = torch.from_numpy(sim.state().copy()).cuda()
        v, rhs, hyp = u.clone(), torch.full_like(u, 7.0), torch.full_like(u, 7.0)
        sim.RHSFunction(rhs, u)
        sim.ApplyBoundaryConditions(v)
        sim.HyperbolicFunction(hyp, v)
        assert torch.equal(u, v) and torch.equal(rhs.isfinite(), hyp.isfinite())
        assert (rhs + hyp).nan_to_num(0.0).abs().max().item() <= 100 * 2.2e-16 * 10 * N
        assert rhs[:9].abs().max().item() == 0.0 and rhs[-9:].abs().max().item() == 0.0


@pytest.mark.parametrize("scheme", ["weno5", "crweno5"])
def test_many_steps_in_several_calls(tmp_path, scheme):
    d = str(tmp_path / "m")
    cases.euler1d_density_wave(d, N=200, n_iter=2100, dt=1e-4, scheme=scheme)
    with Simulation(d) as a, Simulation(d) as b:
        a.time_rk(2100)
        for k in (1, 99, 2000):
            b.time_rk(k)
        assert np.array_equal(a.state(), b.state())
