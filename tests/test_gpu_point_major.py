"""Point-major arrays to planes and back through shared memory, for variable
counts whose stride meets the banks badly (4, 11, 18, 32) and point counts
around a block's: states survive set_state / state bit for bit, the interior
comes back in op-file order, and a boundary fill or a right-hand side leaves the
interior of a caller's array untouched."""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = 3


@pytest.mark.parametrize("layers", [0, 1, 2, 4])
@pytest.mark.parametrize("N,NY", [(8, 7), (26, 10), (131, 17), (250, 250)])
def test_round_trip(tmp_path, layers, N, NY):
    d = str(tmp_path / "p")
    if layers:
        cases.ns2d_photochem_beam(d, N=N, NY=NY, n_iter=1, dt=1e-4, layers=layers, scheme="weno5",
                                  extra_chem={"z_mm": 1.3 * (layers - 1)} if layers > 1 else None)
    else:
        cases.ns2d_shear_layer(d, N=N, NY=NY, n_iter=1, scheme="weno5")
    nv = 4 + 7 * layers
    with Simulation(d) as sim:
        u = np.random.default_rng(N).uniform(0.5, 2.0, (NY + 2 * G, N + 2 * G, nv))
        sim.set_state(u.reshape(-1))
        assert np.array_equal(sim.state().reshape(u.shape), u)
        assert np.array_equal(sim.solution().reshape(NY, N, nv), u[G:-G, G:-G])
        t = torch.from_numpy(u).cuda()
        sim.ApplyBoundaryConditions(t.reshape(-1))
        got = t.cpu().numpy()
        assert np.array_equal(got[G:-G, G:-G], u[G:-G, G:-G])
        assert np.array_equal(got[:G, :G], u[:G, :G]) and np.array_equal(got[-G:, -G:], u[-G:, -G:])   # corners
        assert np.array_equal(got[G:-G, :G], u[G:-G, -2 * G:-G])                                       # periodic in x
        w, r = t.clone(), torch.empty_like(t)
        sim.RHSFunction(r.reshape(-1), w.reshape(-1))
        assert torch.equal(w, t)
