"""Radial grids of more nodes than 16 bits can number: forces, orbits and actions from the cells against the
node form of the same grid (reached as in test_cells_gpu)."""
import numpy as np
import pytest

from test_cells_gpu import padded

pytestmark = pytest.mark.gpu


def coefficients(n):
    """an axisymmetric potential of l = 0, 2, 4 terms in closed form on n radii"""
    r = np.geomspace(1e-3, 1e3, n)
    P, D = np.zeros((25, n)), np.zeros((25, n))
    P[0], D[0] = -1 / (1 + r), 1 / (1 + r) ** 2
    for l, a in ((2, 0.1), (4, -0.02)):
        P[l * (l + 1)] = a * r ** 2 / (1 + r) ** 5
        D[l * (l + 1)] = a * r * (2 - 3 * r) / (1 + r) ** 6
    return r, P, D


@pytest.mark.parametrize("n", [65536, 70001])
def test_more_than_65535_nodes(n):
    import agama_b200
    r, P, D = coefficients(n)
    p = agama_b200.Potential(radii=r, Phi=P, dPhi=D)
    nodes = agama_b200.Potential(radii=r, Phi=padded(P), dPhi=padded(D))
    assert p.info()["gridSizeR"] == n
    rng = np.random.Generator(np.random.PCG64(6))
    x = rng.standard_normal((5000, 3))
    x *= np.exp(rng.uniform(np.log(2e-3), np.log(5e2), (5000, 1))) / np.linalg.norm(x, axis=1)[:, None]
    # the bounds of test_cells_gpu
    phi, acc = p.eval(x, pot=True, acc=True)
    phi0, acc0 = nodes.eval(x, pot=True, acc=True)
    assert np.all(np.abs(phi - phi0) <= 1e-13 * np.abs(phi0))
    assert np.all(np.abs(acc - acc0) <= 3e-12 * (np.abs(phi0) / np.linalg.norm(x, axis=1))[:, None])
    w = np.concatenate([x, rng.standard_normal(x.shape) * 0.3 * np.sqrt(-phi0)[:, None]], 1)[:300]
    T = np.linalg.norm(w[:, :3], axis=1) / np.sqrt(-phi0[:300])
    # (over a fraction of a period an orbit amplifies the difference of the forces by a small factor)
    assert np.allclose(agama_b200.orbit(p, w, T), agama_b200.orbit(nodes, w, T), rtol=1e-7, atol=1e-12)
    fd = 0.5 * np.linalg.norm(w[:, :3], axis=1)
    J, J0 = agama_b200.actions(p, w, fd), agama_b200.actions(p, w, fd, angles=True)[0]
    # (the bound of test_axis_actions_gpu)
    assert np.all(np.abs(J - J0) <= 1e-11 * np.abs(J0).max(1)[:, None])
