"""A grid of more rows of tiles than a launch has in one dimension (65535 rows of
14 points; the last row of tiles is beyond it): the right-hand side of a state
that repeats every 70 rows is, away from both ends, that of a short grid with
the same spacing, tile for tile the same operations: an ulp of the interface
fluxes (below 4) over the spacing (1/64), with a margin of ten: 64 x 4 x 10 x
2.2e-16 = 6e-13.
"""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases, deck

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
Z = deck.BoundaryZone
BIG = 1e99
PERIOD = 70


def rhs(path, NY, pattern, rk="ssprk3"):
    """Right-hand side and the state's rows after a step, interior rows [NY, N, 4]."""
    N = pattern.shape[1] - 6
    zones = [Z("periodic", 0, 1, [0, 0, -BIG, BIG]), Z("periodic", 0, -1, [0, 0, -BIG, BIG]),
             Z("extrapolate", 1, 1, [-BIG, BIG, 0, 0]), Z("extrapolate", 1, -1, [-BIG, BIG, 0, 0])]
    cases.ns2d_channel(path, zones, N=N, NY=NY, L=(N / 64, NY / 64), n_iter=1, dt=1e-3, par="2", Re=-1.0,
                       time_scheme_type=rk)
    rows = (np.arange(NY + 6) - 3) % PERIOD
    with Simulation(path) as sim:
        u = torch.from_numpy(pattern).cuda()[torch.from_numpy(rows).cuda()].contiguous()
        r = torch.full_like(u, 7.0)
        sim.RHSFunction(r.reshape(-1), u.reshape(-1))
        sim.set_state(u.cpu().numpy().reshape(-1))
        sim.time_rk(1)
        return r[3:-3, 3:-3].cpu().numpy(), sim.solution().reshape(NY, N, 4)


def test_rows_beyond_one_dimension(tmp_path):
    rng = np.random.default_rng(5)
    N = 4
    y, x = np.meshgrid(np.arange(PERIOD), np.arange(N + 6) - 3, indexing="ij")
    w = lambda a: a * np.sin(2 * np.pi * (y / PERIOD) + rng.uniform(0, 6)) * np.cos(2 * np.pi * x / N + rng.uniform(0, 6))  # noqa: E731
    rho, u, v, p = 1 + w(0.1), w(0.2), 0.1 + w(0.2), (1 + w(0.1)) / 1.4
    pattern = np.ascontiguousarray(np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], axis=-1))
    periods = 13143                                # 920,010 rows, 65,715 rows of tiles
    for got, want in zip(rhs(str(tmp_path / "tall"), periods * PERIOD, pattern),
                         rhs(str(tmp_path / "short"), 5 * PERIOD, pattern)):
        assert np.abs(want).max() > 0.01
        middle, tall = want[2 * PERIOD:3 * PERIOD], got.reshape(periods, PERIOD, N, 4)
        assert np.abs(tall[1:-1] - middle).max() <= 6e-13
        assert np.abs(tall[0] - want[:PERIOD]).max() <= 6e-13 and np.abs(tall[-1] - want[-PERIOD:]).max() <= 6e-13
