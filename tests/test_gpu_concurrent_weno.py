"""The y pass on its own stream for the explicit schemes (component and
characteristic): the same steps as on one stream, bit for bit."""
import os

import numpy as np
import pytest

from piafs_b200 import Simulation, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interp,chem", [("components", True), ("components", False), ("characteristic", False)])
@pytest.mark.parametrize("scheme", ["weno5", "upw5"])
def test_two_streams_equal_one(tmp_path, interp, chem, scheme):
    d = str(tmp_path / "c")
    if chem:
        cases.ns2d_photochem_beam(d, N=70, NY=45, n_iter=6, dt=0.4 / 2048, scheme=scheme, interp=interp)
    else:
        cases.ns2d_shear_layer(d, N=70, NY=45, n_iter=6, scheme=scheme, interp=interp)
    out = []
    for flag in ("0", "1"):
        old = os.environ.get("PIAFS_GPU_NO_CONCURRENT_Y")
        os.environ["PIAFS_GPU_NO_CONCURRENT_Y"] = flag
        try:
            with Simulation(d) as sim:
                sim.time_rk(6)
                out.append(sim.state())
        finally:
            if old is None:
                del os.environ["PIAFS_GPU_NO_CONCURRENT_Y"]
            else:
                os.environ["PIAFS_GPU_NO_CONCURRENT_Y"] = old
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
