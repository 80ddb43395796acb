"""Kernels that collect the cells around the interface (bulk_then_cells): bit
for bit the oracle's at ragged edges of the 32 x 8 tiles, with one and with
four planes per block and a remainder, from fields that are all bulk, all
interface, and mixed, with a -0 and values just off 0 and 1 among them."""
import numpy as np
import pytest

import oracle.oracle as oo

pytestmark = pytest.mark.gpu

SHAPES = [(6, 6, 6), (35, 11, 9), (133, 75, 136)]


def _field(shape, kind):
    r = np.random.default_rng(7)
    if kind == "bulk":
        return np.ones(shape)
    if kind == "band":
        return r.uniform(0.01, 0.99, size=shape)
    g = np.indices(shape)
    s = sum(((x - 0.45 * n) / (0.4 * n)) ** 2 for x, n in zip(g, shape))
    cc = np.where(s < 0.8, 1.0, np.where(s > 1.0, 0.0, r.uniform(0.0, 1.0, size=shape)))
    cc[tuple(n // 2 for n in shape)] = 1.0 - 2.0 ** -53
    cc[1, 2, 3] = -0.0
    cc[2, 2, 2] = 5e-324
    return cc


@pytest.mark.parametrize("kind", ["bulk", "band", "drop"])
@pytest.mark.parametrize("shape", SHAPES)
def test_filter_and_coefficients(gpu_lib, shape, kind):
    K = gpu_lib.kernels
    cc = _field(shape, kind)
    r = np.random.default_rng(3)
    out0 = r.standard_normal(shape)
    d = K.to_device(out0)
    K.filterc27(K.to_device(cc), d, shape)
    assert np.array_equal(K.to_host(d, shape), oo.filterc27(cc, out0))
    init = [r.standard_normal(shape) for _ in range(4)]
    r1, r2 = 0.5 * (1.0 - 0.0012), 0.0012
    outs = [K.to_device(x) for x in init]
    K.abcei(*outs, K.to_device(cc), r1, r2, shape)
    for o, ref in zip(outs, oo.abcei(cc, r1, r2, init=init)):
        assert np.array_equal(K.to_host(o, shape), ref)


@pytest.mark.parametrize("shape", [(34, 20, 28), (132, 44, 100)])
def test_heights(gpu_lib, shape):
    """Within 1e-12 (pow of the triangle case)."""
    dsg = gpu_lib
    from oracle import Oracle
    inp = dsg.config.droplet(shape[0], impact_speed=3.0).replace(surfacet=5, hswitch=1)
    inp = inp.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2)
    ora = Oracle(inp.as_dict())
    ora.step(1)
    gpu = dsg.Solver(inp, init=False)
    gpu.set_field("cc", ora.field("cc"))
    gpu.calch3d()
    for name in ("hxmin", "hxmax", "hymin", "hymax", "hzmin", "hzmax"):
        assert np.max(np.abs(gpu.field(name) - ora.field(name))) <= 1e-12, name
