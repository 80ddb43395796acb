"""vofmethod called by itself: the flux arrays of its last sweep (ei, res and rhs,
the scratch that the reference passes) are the oracle's, empty cells and the
faces of bc_flux included, whatever the arrays held before, in each sweep order
and on rows that end raggedly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(6, 6, 6), (33, 34, 9), (34, 7, 66), (72, 8, 6)])
def test_fluxes_match_oracle(gpu_lib, shape):
    dsg = gpu_lib
    from oracle import Oracle
    n = [m - 2 for m in shape]
    inp = dsg.config.droplet(n[0] if n[0] % 2 == 0 else n[0] + 1).replace(nx=shape[0], ny=shape[1], nz=shape[2])
    ora, gpu = Oracle(inp.as_dict()), dsg.Solver(inp)
    r = np.random.default_rng(shape[0])
    cc = np.zeros(shape)
    cc[1:-1, 1:-1, 1:-2] = np.where(r.random(tuple(n[:2]) + (n[2] - 1,)) < 0.2, r.random(tuple(n[:2]) + (n[2] - 1,)), 0.0)
    cc[2:4, 2:5, 2:4] = 1.0
    fields = {"cc": cc, "u": r.uniform(-1, 1, shape), "v": r.uniform(-1, 1, shape), "w": r.uniform(-1, 1, shape),
              "ei": r.random(shape), "res": r.random(shape), "rhs": r.random(shape)}
    for name, f in fields.items():
        f = np.asfortranarray(f)
        ora.field(name)[...] = f
        gpu.set_field(name, f)
    for x in (ora, gpu):
        s = x.scalars()
        s.tau, s.tauh = 0.3 * s.h, 0.3
        x.set_scalars(s)
    for _ in range(3):  # the three sweep orders
        ora.vofmethod()
        gpu.vofmethod()
        for name in ("ei", "res", "rhs"):
            # volumes of at most a cell; libm's pow, acos and cos differ by ulps
            assert np.abs(gpu.field(name) - ora.field(name)).max() <= 1e-10, name
    gpu.close()
