"""Boundary zones applied in one launch: zones that overlap (the later zone's
values stay) and grids narrower than the ghost layers (a zone's source can be
another zone's ghost) must give what applying the deck's zones one after
another gives.  Copies and sign changes only: equal bit for bit."""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases, deck

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BIG = 1e99
G = 3
Z = deck.BoundaryZone


def one_after_another(u, zones, x, y):
    """The zones in the deck's order on [row, column, variable] with ghosts."""
    N = (len(x), len(y))
    for z in zones:
        idx = []
        for d, c in ((0, x), (1, y)):
            if d == z.dim:
                b = np.arange(G)
                dst = b - G if z.face == 1 else N[d] + b
                src = b + N[d] - G if z.face == 1 else b
                if z.bctype != "periodic":
                    src = G - 1 - b if z.face == 1 else N[d] - b - 1
                idx.append((dst + G, src + G))
            else:
                lo, hi = z.extent[2 * d], z.extent[2 * d + 1]
                i = np.nonzero((c >= lo) & (c <= hi))[0]
                idx.append((i + G, i + G))
        (dx, sx), (dy, sy) = idx
        v = u[np.ix_(sy, sx)].copy()
        if z.bctype == "reflect":
            v = -v
        elif z.bctype == "dirichlet":
            v[:] = z.values
        u[np.ix_(dy, dx)] = v
    return u


OVERLAP = [Z("extrapolate", 0, 1, [0, 0, -BIG, 0.61]), Z("reflect", 0, 1, [0, 0, 0.39, BIG]),
           Z("dirichlet", 0, -1, [0, 0, 0.5, BIG], values=[1.5, -0.25, 0.5, 3.0]),
           Z("extrapolate", 0, -1, [0, 0, -BIG, BIG]), Z("reflect", 1, 1, [-BIG, BIG, 0, 0]),
           Z("extrapolate", 1, -1, [-BIG, 0.3, 0, 0]), Z("reflect", 1, -1, [0.2, BIG, 0, 0])]
PLAIN = [Z("periodic", 0, 1, [0, 0, -BIG, BIG]), Z("periodic", 0, -1, [0, 0, -BIG, BIG]),
         Z("extrapolate", 1, 1, [-BIG, BIG, 0, 0]), Z("reflect", 1, -1, [-BIG, BIG, 0, 0])]


@pytest.mark.parametrize("zones,N,NY", [(OVERLAP, 20, 13), (PLAIN, 37, 29), (PLAIN, 200, 2), (OVERLAP, 131, 40)])
def test_zones_in_one_launch(tmp_path, zones, N, NY):
    d = str(tmp_path / "z")
    cases.ns2d_channel(d, zones, N=N, NY=NY, n_iter=1, par="2")
    rng = np.random.default_rng(N + NY)
    u = rng.uniform(0.5, 2.0, (NY + 2 * G, N + 2 * G, 4))
    x, y = (np.arange(N) + 0.5) / N, (np.arange(NY) + 0.5) / NY
    want = one_after_another(u.copy(), zones, x, y)
    with Simulation(d) as sim:
        t = torch.from_numpy(u).cuda().contiguous()
        sim.ApplyBoundaryConditions(t.reshape(-1))
        assert np.array_equal(t.cpu().numpy(), want)
