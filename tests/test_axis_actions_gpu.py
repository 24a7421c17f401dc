"""Actions of stars on the z axis above the focus, and so close to it that nu rounds to Delta^2: the
branch of F through such a star lies on the axis, for every focal distance.  The plain request (from the cells
where the potential has them) against the request with angles (from the node form)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 400


@pytest.mark.parametrize("lmax", [12, 2])                   # with cells, and without
@pytest.mark.parametrize("offset", [0, 1e-12, 1e-10, 1e-6])         # R / r
@pytest.mark.parametrize("horizontal", [False, True])       # at a turning point of the lambda motion
def test_axis(lmax, offset, horizontal):
    import torch
    import agama_b200
    from agama_b200.workloads import CONFIG_POTENTIALS
    p = agama_b200.Potential(type="Multipole", **dict(CONFIG_POTENTIALS[5], lmax=lmax))
    rng = np.random.Generator(np.random.PCG64(31))
    fd = rng.uniform(0.05, 3, N)
    w = np.zeros((N, 6))
    w[:, 2] = fd * np.exp(rng.uniform(0.1, 3, N)) * rng.choice([-1, 1], N)
    w[:, 0] = offset * np.abs(w[:, 2])
    v = rng.standard_normal((N, 3))
    v *= (np.sqrt(-2 * p.potential(w[:, :3])) * rng.uniform(0.1, 0.8, N) / np.linalg.norm(v, axis=1))[:, None]
    if horizontal:
        v[:, 1:] = 0
    w[:, 3:] = v
    points, focal = torch.tensor(w, device="cuda"), torch.tensor(fd, device="cuda")
    plain = agama_b200.actions(p, points, fd=focal).cpu().numpy()
    angles = agama_b200.actions(p, points, fd=focal, angles=True)[0].cpu().numpy()
    # the two forms run the same searches on functions that differ by some hundred ulps; the actions
    # are stationary in the limits
    assert np.all(np.abs(plain - angles) <= 1e-11 * np.abs(angles).max(1)[:, None])
