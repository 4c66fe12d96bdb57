"""WENO5 on the characteristic variables of 2D Navier-Stokes, whose projections
are formed in closed form, against the eigenvector matrices of
navierstokes2d.h:194-313 written out in extended precision, in both directions
and for both biases, on grids around one block of interfaces.

Tolerance: a projection is a sum of a few terms of the size of the state (below 4)
over a^2 (above 0.8), and the way back multiplies by the enthalpy (below 4): 4 x 4
x 10 operations x 1.1e-16 = 2e-14; the weights move by 4 d (1e-15) / (d^2 + 1e-6) of a
candidate spread d, below 4e-15.  With a margin of ten: 2e-13.
"""
import numpy as np
import pytest

from piafs_b200 import Simulation, cases

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
G, GAMMA, EPS = 3, 1.4, 1e-6


def matrices(ul, ur, d):
    """L, R [.., 4, 4] of the Roe average of the states ul, ur [.., 4]."""
    def side(u):
        vx, vy = u[..., 1] / u[..., 0], u[..., 2] / u[..., 0]
        p = (u[..., 3] - u[..., 0] * (vx * vx + vy * vy) / 2) * (GAMMA - 1)
        return vx, vy, (u[..., 3] + p) / u[..., 0], np.sqrt(u[..., 0])
    (xl, yl, hl, tl), (xr, yr, hr, tr) = side(ul), side(ur)
    vx, vy, h = [(tl * a + tr * b) / (tl + tr) for a, b in ((xl, xr), (yl, yr), (hl, hr))]
    ek = (vx * vx + vy * vy) / 2
    g1 = GAMMA - 1
    a2 = g1 * (h - ek)
    a = np.sqrt(a2)
    un, ut = (vx, vy) if d == 0 else (vy, vx)
    n, t = (1, 2) if d == 0 else (2, 1)
    L = np.zeros(ul.shape[:-1] + (4, 4), dtype=ul.dtype)
    R = np.zeros_like(L)
    for k, s in ((0, -1), (1, 1)):
        L[..., k, 0] = (g1 * ek - s * a * un) / (2 * a2)
        L[..., k, 1], L[..., k, 2], L[..., k, 3] = -g1 * vx / (2 * a2), -g1 * vy / (2 * a2), g1 / (2 * a2)
        L[..., k, n] += s * a / (2 * a2)
        R[..., 0, k], R[..., 1, k], R[..., 2, k], R[..., 3, k] = 1, vx, vy, h + s * a * un
        R[..., n, k] += s * a
    L[..., 2, 0], L[..., 2, 1], L[..., 2, 2], L[..., 2, 3] = 1 - g1 * ek / a2, g1 * vx / a2, g1 * vy / a2, -g1 / a2
    R[..., 0, 2], R[..., 1, 2], R[..., 2, 2], R[..., 3, 2] = 1, vx, vy, ek
    L[..., 3, 0], L[..., 3, t] = -ut, 1
    R[..., t, 3], R[..., 3, 3] = 1, ut
    return L, R


def weno5(c):
    """The left-biased value of the five cells c[0..4]."""
    b = [13 / 12 * (c[k] - 2 * c[k + 1] + c[k + 2]) ** 2 for k in range(3)]
    b[0] = b[0] + (c[0] - 4 * c[1] + 3 * c[2]) ** 2 / 4
    b[1] = b[1] + (c[1] - c[3]) ** 2 / 4
    b[2] = b[2] + (3 * c[2] - 4 * c[3] + c[4]) ** 2 / 4
    w = [x / (y + EPS) ** 2 for x, y in zip((1 / np.longdouble(10), 6 / np.longdouble(10), 3 / np.longdouble(10)), b)]
    q = [(2 * c[0] - 7 * c[1] + 11 * c[2]) / 6, (-c[1] + 5 * c[2] + 2 * c[3]) / 6, (2 * c[2] + 5 * c[3] - c[4]) / 6]
    return sum(x * y for x, y in zip(w, q)) / sum(w)


def want_values(u, f, d, upw):
    """Interface values of f [W1, W0, 4] with the fields of u along dimension d."""
    ax = 1 - d
    u, f = np.moveaxis(u.astype(np.longdouble), ax, 0), np.moveaxis(f.astype(np.longdouble), ax, 0)
    o = slice(G, u.shape[1] - G)
    n = u.shape[0] - 2 * G + 1
    L, R = matrices(u[G - 1:G - 1 + n, o], u[G:G + n, o], d)
    w = [np.einsum("...vk,...k->...v", L, f[r:r + n, o]) for r in range(6)]
    v = weno5(w[:5]) if upw > 0 else weno5(w[:0:-1])
    return np.moveaxis(np.einsum("...kv,...v->...k", R, v), 0, ax)


@pytest.mark.parametrize("kind", ["flow", "rest"])
@pytest.mark.parametrize("N,NY", [(9, 8), (33, 29), (127, 5)])
def test_values(tmp_path, N, NY, kind):
    d = str(tmp_path / "d")
    cases.ns2d_shear_layer(d, N=N, NY=NY, n_iter=1, scheme="weno5", interp="characteristic")
    rng = np.random.default_rng(N)
    r = lambda a: a * rng.uniform(-1, 1, (NY + 2 * G, N + 2 * G))  # noqa: E731
    a = 0.3 if kind == "flow" else 1e-6
    rho, vx, vy, p = 1 + r(a), r(a), r(a), (1 + r(a)) / GAMMA
    u = np.stack([rho, rho * vx, rho * vy, p / (GAMMA - 1) + rho * (vx * vx + vy * vy) / 2], axis=-1)
    with Simulation(d) as sim:
        t = torch.from_numpy(u).cuda().reshape(-1)
        for dim in (0, 1):
            v = (vx, vy)[dim][..., None]
            f = u * v
            f[..., 1 + dim] += p
            f[..., 3] += p * v[..., 0]
            tf = torch.from_numpy(f).cuda().reshape(-1)
            for upw in (1, -1):
                for uflag, src, arr in ((1, t, u), (0, tf, f)):
                    want = want_values(u, arr, dim, upw)
                    got = torch.zeros(want.size, dtype=torch.float64, device="cuda")
                    sim.InterpolateInterfacesHyp(got, src, t, upw, dim, uflag)
                    err = np.abs(got.cpu().numpy().reshape(want.shape) - want).max()
                    assert err <= 2e-13, (dim, upw, uflag, float(err))
