"""The two forms of the 2-D spline evaluation, from the cells' coefficients (up to eight azimuthal
harmonics) and from the node values (more of them), give the same potential, force, force
derivatives and density: at cell edges, on the axis, in the equatorial plane and at the ends of the
radial grid.

The node form is reached by terms of relative size 1e-40 in every azimuthal order of the largest l,
which add nothing to any value in FP64 and leave the grids as they are.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def coefficients(name):
    import agama_b200
    from agama_b200.workloads import CONFIG_POTENTIALS
    p = dict(CONFIG_POTENTIALS[{"triaxial": 1, "disk": 2, "bar": 3, "galaxy": 5}[name]])
    return agama_b200.multipole_coefs_from_density(p.pop("density"), **p)


def padded(P):
    """the same terms, with negligible ones in the empty places of the largest l"""
    out = P.copy()
    l = int(round(np.sqrt(len(P)))) - 1
    for m in range(-l, l + 1):
        if not out[l * (l + 1) + m].any():
            out[l * (l + 1) + m] = 1e-40 * P[0]
    return out


def points(r, n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    radii = np.concatenate([r[1:-1], r[1:-1] * (1 - 1e-15), r[1:-1] * (1 + 1e-12), r[[0, -1]] * [1.0001, 0.9999],
                            np.exp(rng.uniform(np.log(r[0]), np.log(r[-1]), size=n))])
    radii = radii[(radii > r[0] * (1 + 1e-5)) & (radii < r[-1] * (1 - 1e-5))]
    ct = np.concatenate([[1, -1, 0, 1 - 1e-12, -1 + 1e-12, 1e-13, -1e-13], rng.uniform(-1, 1, size=9)])
    phi = np.concatenate([[0, np.pi / 2, np.pi], rng.uniform(-np.pi, np.pi, size=4)])
    ct, phi = rng.choice(ct, size=len(radii)), rng.choice(phi, size=len(radii))
    st = np.sqrt((1 - ct) * (1 + ct))
    return radii[:, None] * np.stack([st * np.cos(phi), st * np.sin(phi), ct], 1)


@pytest.mark.parametrize("name", ["triaxial", "bar", "disk", "galaxy"])
@pytest.mark.parametrize("n", [1, 127, 129, 5000])
def test_cells_against_nodes(name, n):
    import agama_b200
    r, P, D = coefficients(name)
    cells = agama_b200.Potential(radii=r, Phi=P, dPhi=D)
    nodes = agama_b200.Potential(radii=r, Phi=padded(P), dPhi=padded(D))
    assert nodes.info()["mmax"] == nodes.info()["lmax"] == cells.info()["lmax"]
    assert nodes.info()["gridSizeTau"] == cells.info()["gridSizeTau"]
    x = points(r, n, 7)
    rr = np.linalg.norm(x, axis=1)
    phi1, acc1, h1 = cells.eval(x, pot=True, acc=True, der=True)
    phi2, acc2, h2 = nodes.eval(x, pot=True, acc=True, der=True)
    # both forms interpolate the same node data, each with rounding errors of some hundred ulps of the
    # cell's values per order of derivative (a cell's width in tau enters as ~1/30 per order)
    scale = np.abs(phi2)
    assert np.all(np.abs(phi1 - phi2) <= 1e-13 * scale)
    assert np.all(np.abs(acc1 - acc2) <= 3e-12 * (scale / rr)[:, None])
    # next to the axis a rounding error of some ulps of a harmonic m enters the second derivative over
    # the azimuth as m^2 / R^2 (the node form's harmonics do not vanish exactly towards the upper pole)
    R = np.hypot(x[:, 0], x[:, 1])
    off = R > 1e-6 * rr                             # on the axis the phi derivatives are degenerate
    mmax = cells.info()["mmax"]
    bound = ((1e-9 + 4 * np.finfo(float).eps * mmax ** 2 * (rr / np.maximum(R, 1e-300)) ** 2) * scale / rr ** 2)[off]
    assert np.all(np.abs(h1 - h2)[off] <= bound[:, None])
    rho1, rho2 = cells.density(x), nodes.density(x)
    assert np.all(np.abs(rho1 - rho2)[off] <= bound)
