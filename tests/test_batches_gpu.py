"""Actions, angles and orbits of a point do not depend, to the bit, on the batch that it comes in: the work
queues hand the points out in claims (16 points of the integrals, 8 idle lanes of the root searches, one
orbit a group of lanes), so batches on both sides of a claim, a warp and a block are cut from a larger one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 7, 8, 9, 15, 16, 17, 31, 33, 127, 129, 513]


def stars(n):
    rng = np.random.Generator(np.random.PCG64(5))
    x = rng.standard_normal((n, 3)) * np.exp(rng.uniform(-2, 2, (n, 1)))
    v = rng.standard_normal((n, 3)) * 0.3
    return np.concatenate([x, v], 1)


@pytest.fixture(scope="module")
def setup():
    import torch
    import agama_b200
    from test_cells_gpu import coefficients
    r, P, D = coefficients("disk")
    pot = agama_b200.Potential(radii=r, Phi=P, dPhi=D)
    w = stars(1500)
    phi = pot.potential(np.ascontiguousarray(w[:, :3]))
    w[:, 3:] *= np.sqrt(np.maximum(-phi, 0))[:, None]       # bound orbits
    points = torch.tensor(w, device="cuda")
    af = agama_b200.ActionFinder(pot)
    return pot, af, points


def same(a, b):
    return np.array_equal(a.cpu().numpy(), b.cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("n", SIZES)
def test_actions_and_angles(setup, n):
    pot, af, points = setup
    want, (J, theta, Omega) = af(points), af(points, angles=True, frequencies=True)
    first = 1500 - n
    assert same(af(points[first:]), want[first:])
    J1, theta1, Omega1 = af(points[first:], angles=True, frequencies=True)
    assert same(J1, J[first:]) and same(theta1, theta[first:]) and same(Omega1, Omega[first:])


@pytest.mark.parametrize("n", [1, 3, 31, 33, 129])
def test_orbits(setup, n):
    import agama_b200
    pot, af, points = setup
    want = agama_b200.orbit(pot, points[:200], 3.0)
    assert same(agama_b200.orbit(pot, points[200 - n:200], 3.0), want[200 - n:])
