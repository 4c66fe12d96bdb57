"""A step that sums the residual norm gives the state of one that does not, bit
for bit (the printing interval must not change a solution file), and the norm
is that of the step's change: a sum of squares in another order, 1e-12
relative.
"""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases

pytestmark = pytest.mark.gpu


def line(scheme, upw, N):
    return lambda d: cases.euler1d_density_wave(d, N=N, n_iter=4, dt=0.1 / N, scheme=scheme, upwinding=upw)


def shear(scheme, upw, N, NY, **kw):
    return lambda d: cases.ns2d_shear_layer(d, N=N, NY=NY, n_iter=4, scheme=scheme, upwinding=upw, **kw)


def chem(scheme, upw, N, NY, **kw):
    return lambda d: cases.ns2d_photochem_beam(d, N=N, NY=NY, n_iter=4, dt=0.4 / 2048, scheme=scheme, upwinding=upw,
                                               flow=(0.2, 0.1), noise=1e-2, **kw)


DECKS = {"1d-roe": line("weno5", "roe", 1024), "1d-llf": line("weno5", "llf-char", 100), "1d-8": line("weno5", "roe", 8),
         "1d-compact": line("crweno5", "roe", 600), "1d-compact-two-warps": line("crweno5", "rusanov", 6001),
         "shear": shear("crweno5", "llf-char", 33, 29), "shear-one-stage": shear("weno5", "roe", 33, 29, time_scheme_type="1fe"),
         "shear-past-148-tiles": shear("weno5", "rf-char", 300, 217, dt=2e-4), "chem": chem("weno5", "roe", 64, 64),
         "chem-past-148-tiles": chem("crweno5", "llf-char", 200, 230), "chem-two-layers": chem("weno5", "llf-char", 40, 33, layers=2, extra_chem={"z_mm": 1.3}),
         "chem-44": chem("crweno5", "rusanov", 33, 29, time_scheme_type="44")}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", DECKS)
def test_state_does_not_depend_on_the_norm(tmp_path, name, precision):
    d = str(tmp_path / "d")
    DECKS[name](d)
    with Simulation(d, precision) as a, Simulation(d, precision) as b:
        norms, changes = [], []
        for _ in range(3):
            before = b.solution()
            norms.append(b.time_rk_norm(1))
            changes.append(np.sqrt(((b.solution() - before) ** 2).sum() / (b.info["dim"][0] * b.info["dim"][1])))
        a.time_rk(3)
        assert np.isfinite(a.state()).all() and np.array_equal(a.state(), b.state())
        assert a.info["t"] == b.info["t"] and a.info["iter"] == b.info["iter"]
        assert np.allclose(norms, changes, rtol=1e-12, atol=0.0)
        assert np.isclose(a.time_rk_norm(2), b.time_rk_norm(2), rtol=1e-12, atol=0.0)
        a.time_rk(1), b.time_rk(1)
        assert np.array_equal(a.state(), b.state())
