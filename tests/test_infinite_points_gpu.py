"""Forces of axisymmetric potentials at points at infinity: the component along an infinite x or y alone is not
a number, the others are 0 (host and device arrays)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config", [2, 4, 5])
def test_force(config):
    import torch
    import agama_b200
    from agama_b200.workloads import CONFIG_POTENTIALS
    p = agama_b200.Potential(type="Multipole", **CONFIG_POTENTIALS[config])
    finite = [0, 1e-200, 1., -3., 1e200]
    x = np.array([[s * np.inf, a, b] for s in (1, -1) for a in finite for b in finite + [np.inf]])
    for points, axis in ((x, 0), (x[:, [1, 0, 2]], 1)):
        for force in (p.force(points), p.force(torch.tensor(points, device="cuda")).cpu().numpy()):
            assert np.isnan(force[:, axis]).all()
            assert np.all(np.delete(force, axis, 1) == 0)
