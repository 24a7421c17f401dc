"""The acceleration entry point writes minus the gradient (and minus the Hessian where asked) of
agama_evalPotentialManyDevice, to the bit: inside the cells, beyond them, on the axis, at the centre and
at non-finite points, for potentials with and without cells, at the edges of a block."""
import numpy as np
import pytest

from test_cells_gpu import coefficients, padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,nodes", [("triaxial", False), ("bar", False), ("disk", False), ("disk", True)])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 3001])
def test_acceleration_is_minus_the_gradient(name, nodes, n):
    import torch
    import agama_b200
    from agama_b200 import _native, _dev_ptr, _current_stream
    r, P, D = coefficients(name)
    pot = agama_b200.Potential(radii=r, Phi=padded(P) if nodes else P, dPhi=padded(D) if nodes else D)
    rng = np.random.Generator(np.random.PCG64(n))
    x = rng.standard_normal((n, 3)) * np.exp(rng.uniform(np.log(r[0]) - 3, np.log(r[-1]) + 3, (n, 1)))
    x[::7, :2] = 0
    x[3::50] = 0
    x[5::50, 0] = np.nan
    x[6::50, 1] = np.inf
    p = torch.tensor(x, device="cuda")
    phi, grad, hess = (torch.empty(s, dtype=torch.float64, device="cuda") for s in ((n,), (n, 3), (n, 6)))
    only = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    lib = _native.lib()
    _native.check(lib.agama_evalPotentialManyDevice(pot.handle, n, _dev_ptr(p), _dev_ptr(phi), _dev_ptr(grad),
                                                    _dev_ptr(hess), _current_stream()))
    _native.check(lib.agama_evalPotentialManyDevice(pot.handle, n, _dev_ptr(p), None, _dev_ptr(only), None,
                                                    _current_stream()))
    acc, der = pot.forceDeriv(p)
    phi2, acc2, hess2 = pot.eval(p, pot=True, acc=True, der=True)
    for got, want in ((acc, -grad), (der, -hess), (phi2, phi), (acc2, -grad), (hess2, hess), (pot.force(p), -only)):
        assert np.array_equal(got.cpu().numpy(), want.cpu().numpy(), equal_nan=True)
