"""The CRWENO5 line solve at the sizes where its rows, chunks, warps, CTAs and
clusters begin and end, on smooth lines (whose separator couplings decay, so
that the reduction stops early) and on rough ones (random values and jumps,
where the couplings between chunks do not), against the oracle's serial
systems.

Tolerance: both solve the same systems in FP64 with another elimination order.
On smooth data the systems are diagonally dominant (condition number below
10) and the differences a few ulps: 1e-13 of the line's scale, with a margin of
ten.  On rough data a row's off-diagonal can be twice its diagonal where one
weight takes all, and a run of ten such rows amplifies rounding by 2^10: 1e-12,
with a margin of a hundred for longer runs.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle
from piafs_b200 import Simulation, cases

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = [3, 4, 5, 9, 32, 33, 34, 127, 128, 129, 130, 255, 256, 257, 258, 264, 511, 513, 2047, 2048, 2049, 4096, 4097,
         4098, 4099, 6001, 16385, 20011]
G = 3


def line(N, kind):
    rng = np.random.default_rng(N)
    x = np.arange(-G, N + G) / N
    if kind == "smooth":
        u = np.stack([1.0 + 0.2 * np.sin(2 * np.pi * (k + 1) * x + k) for k in range(3)], axis=1)
    else:
        u = rng.uniform(-1.0, 1.0, (N + 2 * G, 3)) + 5.0 * (rng.uniform(size=(N + 2 * G, 1)) > 0.9)
    return np.ascontiguousarray(u)


@pytest.mark.parametrize("weno", ["js", "yc", "borges", "mapped", "none"])
@pytest.mark.parametrize("kind,tol", [("smooth", 1e-12), ("rough", 1e-10)])
def test_lines_of_every_edge_size(tmp_path, kind, tol, weno):
    sizes = SIZES if weno in ("js", "yc") else [4, 129, 513, 4098]
    for N in sizes:
        d = str(tmp_path / f"n{N}")
        key = {"js": None, "none": {"no_limiting": 1}}.get(weno, {weno: 1})
        cases.euler1d_density_wave(d, N=N, n_iter=1, scheme="crweno5", weno=key)
        case = oracle.load(d)
        u = line(N, kind)
        f = np.ascontiguousarray(u[::-1])
        with Simulation(d) as sim:
            du, df = torch.from_numpy(u).cuda().reshape(-1), torch.from_numpy(f).cuda().reshape(-1)
            for upw in (1, -1):
                for uflag in (1, 0):
                    want = np.zeros((N + 1, 3))
                    oracle.lib().orc_interp(C.byref(case.P), oracle._dp(want), oracle._dp(f), oracle._dp(u), upw, 0,
                                            uflag)
                    got = torch.zeros((N + 1) * 3, dtype=torch.float64, device="cuda")
                    sim.InterpolateInterfacesHyp(got, df, du, upw, 0, uflag)
                    err = np.abs(got.cpu().numpy().reshape(N + 1, 3) - want).max()
                    assert err <= tol * np.abs(u).max(), (N, upw, uflag, err)
