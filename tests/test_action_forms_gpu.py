"""Actions of the plain request (phase 1 and searches from the cells, fudge.cuh) and of the request with angles
(the same steps from the node form, fudge_nodes.cuh) for the same points, through both texts of phase 1: generic
stars, stars in and crossing the plane, at turning points of either motion, unbound and undefined ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stars(p, n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.standard_normal((n, 3)) * np.array([1, 1, 0.4]) * np.exp(rng.uniform(-2, 3, (n, 1)))
    v = rng.standard_normal((n, 3))
    v *= (np.sqrt(-2 * p.potential(x)) * rng.uniform(0.1, 0.95, n) / np.linalg.norm(v, axis=1))[:, None]
    kind = np.arange(n) % 8
    x[kind == 1, 2] = 0                             # in the plane
    planar = kind == 2                              # ... and staying there
    x[planar, 2] = v[planar, 2] = 0
    for k in (3, 4):                                # no radial velocity; none along z either
        c, s = x[kind == k, :2].T / np.hypot(*x[kind == k, :2].T)
        vt = -v[kind == k, 0] * s + v[kind == k, 1] * c
        v[kind == k, 0], v[kind == k, 1] = -vt * s, vt * c
    v[kind == 4, 2] = 0
    v[kind == 5] *= 20                              # unbound
    w = np.concatenate([x, v], 1)
    w[6::64, 0] = np.nan
    w[14::64, 3] = np.inf
    w[22::64] = 0
    return w


@pytest.mark.parametrize("config,lmax", [(2, 8), (4, 6), (5, 12), (5, 2)])
@pytest.mark.parametrize("finder", [True, False])
def test_same_actions(config, lmax, finder):
    import torch
    import agama_b200
    from agama_b200.workloads import CONFIG_POTENTIALS
    p = agama_b200.Potential(type="Multipole", **dict(CONFIG_POTENTIALS[config], lmax=lmax))
    w = stars(p, 4096, config)
    points = torch.tensor(w, device="cuda")
    if finder:
        af = agama_b200.ActionFinder(p)
        plain, angles = af(points), af(points, angles=True)[0]
    else:
        fd = torch.tensor(0.4 * np.linalg.norm(np.nan_to_num(w[:, :3]), axis=1) + 0.05, device="cuda")
        plain, angles = agama_b200.actions(p, points, fd=fd), agama_b200.actions(p, points, fd=fd, angles=True)[0]
    plain, angles = plain.cpu().numpy(), angles.cpu().numpy()
    assert np.array_equal(np.isnan(plain), np.isnan(angles))
    ok = ~np.isnan(angles).any(1)
    assert ok.sum() > 3000
    # the bound of test_axis_actions_gpu; a star at a turning point (whether it has a root search there is
    # decided by the sign of a rounding error) may be 1e-10 of its range, FUDGE_MINIMUM_RANGE, off in the limit
    bound = 1e-9 * np.abs(angles[ok]).max(1)[:, None]
    assert np.all(np.abs(plain[ok] - angles[ok]) <= bound)
    generic = ok & np.isin(np.arange(len(w)) % 8, (0, 1, 6, 7)) & (np.linalg.norm(np.nan_to_num(w[:, :3]), axis=1) > 0)
    assert np.all(np.abs(plain[generic] - angles[generic]) <= 1e-11 * np.abs(angles[generic]).max(1)[:, None])
