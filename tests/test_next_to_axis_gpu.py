"""Second derivatives at points so close to the z axis that 1 / R^2 overflows: those at a distance where it
does not (xx, yy and zz in the planes x = 0 and y = 0)."""
import numpy as np
import pytest

from test_cells_gpu import coefficients

pytestmark = pytest.mark.gpu


def points(R):
    return np.array([[c * R, s * R, z] for c, s in ((1, 0), (0, 1), (-1, 0), (0, -1)) for z in (1., -1., 0.25, -4.)])


@pytest.mark.parametrize("name", ["triaxial", "bar", "disk"])
@pytest.mark.parametrize("R", [1e-160, 1e-155, 1e-154, 1e-150])
def test_hessian(name, R):
    import agama_b200
    r, P, D = coefficients(name)
    p = agama_b200.Potential(radii=r, Phi=P, dPhi=D)
    far = points(1e-100)
    phi, want = p.eval(far, pot=True, der=True)
    got = p.eval(points(R), pot=False, der=True)
    # at these heights, whose reciprocals are exact, tau = +-1 and the m != 0 harmonics vanish: rounding, and
    # that of x^2 + y^2 where it is subnormal
    bound = (1e-9 + 8 * 5e-324 / R ** 2) * np.abs(phi) / far[:, 2] ** 2
    assert np.all(np.abs(got - want)[:, :3] <= bound[:, None])
