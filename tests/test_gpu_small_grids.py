"""The kernels' forms for grids of few tiles, on both sides of the sizes where
they end: 148 tiles of 16 x 14 points (592 x 56; 593 x 56 has 152) for the
kernel that ends a stage, 148 blocks of a 32 x 32 tile's parts (90 x 186 has 144
with eleven variables, 90 x 187 168) for the transposed state, against the
oracle's right-hand side.

Tolerance: a few ulps of interface fluxes (below 3) over the spacing, 1/600, with
ten operations: 600 x 3 x 10 x 2.2e-16 = 4e-12 absolute; a margin of thirty for
the compact systems: 1.2e-10.
"""
import numpy as np
import pytest

from oracle import oracle
from piafs_b200 import Simulation
from test_gpu_stage2d import flow, make

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upw,scheme", [("llf-char", "crweno5"), ("roe", "weno5"), ("rf-char", "crweno5"),
                                        ("rusanov", "weno5")])
@pytest.mark.parametrize("chem", [False, True])
@pytest.mark.parametrize("N,NY", [(592, 56), (593, 56), (90, 186), (90, 187)])
def test_right_hand_side(tmp_path, N, NY, upw, chem, scheme):
    d = str(tmp_path / "s")
    make(d, N, NY, upw, chem, scheme)
    case = oracle.load(d)
    u = flow(case, N)
    t = 0.012
    want, _ = case.rhs(u, t)
    with Simulation(d) as sim:
        du = torch.from_numpy(u).cuda()
        r = torch.full_like(du, 7.0)
        sim.RHSFunction(r, du, t)
        assert np.abs(r.cpu().numpy() - want).max() <= 1.2e-10
