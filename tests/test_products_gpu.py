"""FP64 sweeps that share the products of gas cells (and take u itself in liquid
of coefficient 1): bit for bit the oracle's mglin, where both fluids and their
interface lie across warps, rows are no multiple of a warp, and one sweep,
none, or several share the products of the first."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho2", [None, 0.3])
@pytest.mark.parametrize("npre", [0, 1, 4])
@pytest.mark.parametrize("shape", [(48, 48, 48), (96, 48, 52), (52, 76, 60), (140, 36, 44)])
def test_mglin_matches_oracle(gpu_lib, shape, npre, rho2):
    dsg = gpu_lib
    from oracle import Oracle
    inp = dsg.config.droplet(shape[0], impact_speed=2.0)
    inp = inp.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2)
    ora, gpu = Oracle(inp.as_dict()), dsg.Solver(inp)
    if rho2 is not None:  # a coefficient of gas with a full mantissa
        s = ora.scalars()
        s.rho2 = rho2
        ora.set_scalars(s)
    ora.step(1)  # a realistic right-hand side and coefficients
    for name in ("rhs", "a", "b", "c", "ei"):
        gpu.set_field(name, ora.field(name))
    s, so = gpu.scalars(), ora.scalars()
    so.npre, so.npost = npre, max(npre, 1)
    ora.set_scalars(so)
    for f in ("npre", "npost", "ntop", "rho1", "rho2"):
        setattr(s, f, getattr(so, f))
    gpu.set_scalars(s)
    ora.mglin()
    gpu.mglin()
    assert np.array_equal(gpu.field("p"), ora.field("p"))
