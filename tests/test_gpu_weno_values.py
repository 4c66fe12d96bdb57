"""Interface values of explicit WENO5 (Jiang-Shu weights, the difference form
shared by the single-run kernels and the batched tile) against the oracle, on
smooth and rough lines and lines on a large constant background.

Tolerance: a value is a convex combination of candidates, each a sum of a few
cells; rounding moves the candidates by a few ulps of the cells and the weights
by a relative 1e-14 or so of differences between candidates: 1e-14 of the
largest cell, with a margin of ten.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle
from piafs_b200 import Simulation, cases

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G = 3


@pytest.mark.parametrize("kind", ["smooth", "rough", "background", "constant"])
@pytest.mark.parametrize("N", [8, 255, 1024])
def test_values(tmp_path, kind, N):
    rng = np.random.default_rng(N)
    x = np.arange(-G, N + G)[:, None] / N
    u = {"smooth": 1.0 + 0.2 * np.sin(2 * np.pi * x * [1, 2, 3]),
         "rough": rng.uniform(-1, 1, (N + 2 * G, 3)) + 5.0 * (rng.uniform(size=(N + 2 * G, 3)) > 0.9),
         "background": 1e3 + 1e-6 * rng.uniform(-1, 1, (N + 2 * G, 3)),
         "constant": np.full((N + 2 * G, 3), 0.3)}[kind]
    u = np.ascontiguousarray(u)
    d = str(tmp_path / "d")
    cases.euler1d_density_wave(d, N=N, n_iter=1, scheme="weno5")
    case = oracle.load(d)
    with Simulation(d) as sim:
        t = torch.from_numpy(u).cuda().reshape(-1)
        for upw in (1, -1):
            want = np.zeros((N + 1, 3))
            oracle.lib().orc_interp(C.byref(case.P), oracle._dp(want), oracle._dp(u), oracle._dp(u), upw, 0, 1)
            got = torch.zeros((N + 1) * 3, dtype=torch.float64, device="cuda")
            sim.InterpolateInterfacesHyp(got, t, t, upw, 0, 1)
            assert np.abs(got.cpu().numpy().reshape(N + 1, 3) - want).max() <= 1e-13 * np.abs(u).max()
