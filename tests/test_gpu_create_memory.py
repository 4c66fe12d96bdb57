"""The y pass on a stream of its own takes no state array of its own: a 2D
simulation holds as much device memory with it as without (up to what a stream
costs, and the driver's 2 MB granules), for explicit and compact schemes."""
import pytest

from piafs_b200 import Simulation, cases

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def held(d):
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with Simulation(d) as sim:
        sim.time_rk(1)
        return free - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("scheme", ["weno5", "crweno5"])
def test_device_memory(tmp_path, monkeypatch, scheme):
    d = str(tmp_path / "d")
    cases.ns2d_photochem_beam(d, N=1200, NY=500, n_iter=1, dt=1e-4, scheme=scheme)
    state = 1206 * 506 * 11 * 8
    torch.zeros(1, device="cuda")
    held(d)                         # what a process loads once
    both = held(d)
    monkeypatch.setenv("PIAFS_GPU_NO_CONCURRENT_Y", "1")
    assert both - held(d) < state / 4
