"""The ways of asking for steps of a 1D line whose steps run together: waiting,
not waiting, one step from and to the host, with a boundary that ghosts depend
on.  The same launches on the same values: equal bit for bit, ghosts, clock and
step count included."""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases, deck

pytestmark = pytest.mark.gpu
Z = deck.BoundaryZone
WALLS = [Z("slip-wall", 0, 1, [0.0, 0.0], [0.1]), Z("slip-wall", 0, -1, [0.0, 0.0], [0.0])]


@pytest.mark.parametrize("zones", [None, WALLS], ids=["periodic", "walls"])
@pytest.mark.parametrize("scheme,N", [("weno5", 1000), ("crweno5", 600)])
def test_calls_agree(tmp_path, scheme, N, zones):
    d = str(tmp_path / "d")
    dt = 0.1 / N
    cases.euler1d_density_wave(d, N=N, n_iter=5, dt=dt, scheme=scheme, zones=zones)
    with Simulation(d) as a, Simulation(d) as b, Simulation(d) as c:
        assert a.info["launches_per_step"] == 1
        u, t = c.state(), 0.0
        a.time_rk(5)
        b.time_rk_async(2)
        b.time_rk_async(3)
        b.synchronize()
        for _ in range(5):
            u = c.time_rk_host(u, t)
            t += dt
        assert np.isfinite(u).all()
        assert np.array_equal(a.state(), b.state()) and np.array_equal(a.state(), np.asarray(u).reshape(-1))
        assert a.info["t"] == b.info["t"] == c.info["t"] and a.info["iter"] == b.info["iter"] == c.info["iter"] == 5
