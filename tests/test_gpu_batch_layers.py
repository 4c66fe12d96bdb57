"""Batch members of several chemistry layers: every launch shape takes members
of as many layers as its tile has shared memory for (227 KB a CTA, the counts
below at the plain pitch of a row), refuses one layer more, and gives what the
deck gives alone: 1e-12 in FP64, 1e-5 in mixed precision relative to each
variable's largest value, the bars of the other batch tests.
"""
import numpy as np
import pytest

from piafs_b200 import Batch, PiafsError, Simulation, cases

pytestmark = pytest.mark.gpu

# (tile x, tile y, CTAs an SM): layers in FP64, in mixed precision
LAYERS = {(16, 16, 1): (1, 1), (32, 8, 1): (1, 1), (16, 8, 2): (4, 4), (32, 4, 2): (4, 3), (8, 16, 2): (4, 4),
          (16, 15, 1): (1, 2), (32, 7, 1): (1, 2), (16, 7, 2): (4, 4)}


def make(d, layers):
    cases.ns2d_photochem_beam(d, N=39, NY=27, n_iter=3, dt=2e-4, scheme="weno5", noise=1e-2, flow=(0.2, 0.1),
                              layers=layers, extra_chem={"z_mm": 1.3 * (layers - 1)} if layers > 1 else None)
    return d


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", LAYERS, ids=lambda s: f"{s[0]}x{s[1]}")
def test_layers_that_fit(tmp_path, shape, precision):
    most = LAYERS[shape][precision == "mixed"]
    d = make(str(tmp_path / "fits"), most)
    with Simulation(d) as s:
        s.time_rk(3)
        want = s.solution()
    with Batch(precision) as b:
        b.set_launch(*shape)
        i = b.add(d, 3)
        b.step(3)
        got = b.solution(i)
        assert got.shape[1] == 4 + 7 * most
        top = np.maximum(np.abs(want).max(axis=0), 1e-6 * np.abs(want).max())
        assert (np.abs(got - want).max(axis=0) / top).max() <= (1e-12 if precision == "fp64" else 1e-5)
        if most < 4:
            with pytest.raises(PiafsError):
                b.add(make(str(tmp_path / "more"), most + 1), 3)
