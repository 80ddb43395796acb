"""relax and resid keep the reference's bits in every form that the spacing and
omega select (exact products fused or not), with the ghosts written by the
sweep itself: grids whose spacing is and is not a power of two, of one and two
cells along a side, omegas whose 1 - omega is and is not a power of two."""
import numpy as np
import pytest

import oracle.oracle as oo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("omega", [1.5, 1.3, 0.75])
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 3, 5), (7, 9, 11), (34, 6, 4), (67, 5, 10)])
def test_relax_resid_forms(gpu_lib, shape, omega):
    K = gpu_lib.kernels
    r = np.random.default_rng(7)
    u, rhs = r.standard_normal(shape), r.standard_normal(shape)
    a, b, c = (r.uniform(1.0, 833.0, size=shape) for _ in range(3))
    ei = 1.0 / (a + b + c + 1.0)
    du = K.to_device(u)
    dev = [K.to_device(x) for x in (rhs, a, b, c, ei)]
    ref = u
    for _ in range(2):
        ref = oo.relax(ref, 1.0, rhs, a, b, c, ei, omega)
        K.relax(du, 1.0, *dev, shape, omega)
    assert np.array_equal(K.to_host(du, shape), ref)
    res = K.to_device(np.zeros(shape))
    K.resid(1.0, res, du, dev[0], dev[1], dev[2], dev[3], shape)
    assert np.array_equal(K.to_host(res, shape), oo.resid(1.0, ref, rhs, a, b, c))
