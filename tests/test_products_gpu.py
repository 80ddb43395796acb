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


def test_fused_form_is_the_same_in_an_ensemble(gpu_lib):
    """Members keep levels in clusters and passes that a context of its own runs
    as cooperative phases; the short fused form applies to neither."""
    dsg = gpu_lib
    inputs = [dsg.config.droplet(n, mode=1, tol=1e-8, impact_speed=2.0) for n in (32, 40, 48, 64)]
    alone = []
    for inp in inputs:
        with dsg.Solver(inp) as s:
            s.step(1)
            alone.append(s.field("p"))
    with dsg.Ensemble(inputs, workers=2) as e:
        e.step(1)
        for i, p in enumerate(alone):
            assert np.array_equal(e.member(i).field("p"), p), i
