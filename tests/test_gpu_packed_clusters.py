"""Packed interface values on lines that clusters of CTAs solve (4098 interfaces
and more), in either direction, with chemistry and without: the same sums and
differences formed by the solve instead of the upwinding, so equal bit for bit
to the unpacked arrays."""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("chemistry", [False, True])
@pytest.mark.parametrize("upw", ["llf-char", "roe", "rusanov"])
@pytest.mark.parametrize("N,NY", [(4200, 5), (5, 4500)])
def test_packed_equals_unpacked(tmp_path, monkeypatch, N, NY, upw, chemistry, precision):
    d = str(tmp_path / "d")
    cases.ns2d_photochem_beam(d, N=N, NY=NY, n_iter=3, dt=1e-5, upwinding=upw, chemistry=chemistry, noise=1e-2,
                              flow=(0.2, 0.1))
    out = []
    for off in ("0", "1"):
        monkeypatch.setenv("PIAFS_GPU_NO_PACKED_SPECIES", off)
        with Simulation(d, precision) as sim:
            sim.time_rk(3)
            out.append(sim.state())
    assert np.isfinite(out[0]).all() and np.array_equal(*out)
