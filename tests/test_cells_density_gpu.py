"""Densities from the cells and from the node values against the terms that they are the sum of, and the second
derivatives and the density on the z axis (test_cells_gpu bounds the density by the potential, and leaves out
the points within 1e-6 of the axis)."""
import numpy as np
import pytest

from test_cells_gpu import coefficients, padded

pytestmark = pytest.mark.gpu

# Either form rounds a cell's values (up to ~15 in the logarithmic scaling) to 2e-16, and the second derivatives of a
# quintic segment are up to 60 / width^2 times that: widths of ~0.05 in tau, where that is largest, give 8e-11
# of |Phi| / r^2
EPS = 2e-10


def potentials(name):
    import agama_b200
    r, P, D = coefficients(name)
    return r, agama_b200.Potential(radii=r, Phi=P, dPhi=D), agama_b200.Potential(radii=r, Phi=padded(P), dPhi=padded(D))


@pytest.mark.parametrize("name", ["triaxial", "bar", "disk", "galaxy"])
def test_density(name):
    r, cells, nodes = potentials(name)
    rng = np.random.Generator(np.random.PCG64(11))
    n = 20000
    ct, azimuth = rng.uniform(-1, 1, n), rng.uniform(-np.pi, np.pi, n)
    rad = np.exp(rng.uniform(np.log(r[0]) + 1e-3, np.log(r[-1]) - 1e-3, n))
    R = np.maximum(rad * np.sqrt(1 - ct ** 2), 0.02 * rad)
    x = np.stack([R * np.cos(azimuth), R * np.sin(azimuth), rad * ct], 1)
    phi, g, h = nodes.eval_cyl(np.stack([R, x[:, 2], azimuth], 1))
    scale = (np.abs(phi) / (R ** 2 + x[:, 2] ** 2) + np.abs(h[:, 0]) + np.abs(g[:, 0] / R) + np.abs(h[:, 1]) +
             np.abs(h[:, 2]) / R ** 2)
    # (a harmonic m's rounding enters the azimuthal term as m^2 / R^2)
    m = cells.info()["mmax"]
    bound = (EPS + 4 * np.finfo(float).eps * m ** 2 * (rad / R) ** 2) * scale / (4 * np.pi)
    a, b = cells.density(x), nodes.density(x)
    assert np.all(np.abs(a - b) <= bound + 1e-12 * np.abs(b))


@pytest.mark.parametrize("name", ["triaxial", "bar", "disk", "galaxy"])
def test_axis(name):
    r, cells, nodes = potentials(name)
    z = np.exp(np.linspace(np.log(r[0]) + 1e-3, np.log(r[-1]) - 1e-3, 500))
    z = np.concatenate([z, -z])
    points = np.stack([0 * z, z, 0 * z], 1)
    (phi, g1, h1), (_, g2, h2) = cells.eval_cyl(points), nodes.eval_cyl(points)
    scale = np.abs(phi) / z ** 2
    for k in (0, 1, 3):                         # dR2, dz2, dRdz
        assert np.all(np.abs(h1[:, k] - h2[:, k]) <= EPS * scale), k
    if cells.info()["mmax"] == 0:               # (otherwise the axis is the node form's in either potential)
        x = np.stack([0 * z, 0 * z, z], 1)
        for offset in (0, 1e-9):
            x[:, 0] = offset * np.abs(z)
            a, b = cells.density(x), nodes.density(x)
            assert np.all(np.abs(a - b) <= EPS * (scale + 2 * np.abs(h2[:, 0]) + np.abs(h2[:, 1])) / (4 * np.pi) + 1e-12 * np.abs(b))
