"""VOF sweeps over the occupied cells only (vof.cu) against the oracle, where
the bit words and rows of the scan end raggedly: rows of 5, 31, 32, 33 and 70
cells, liquid at every face, isolated cells, values that are full, empty,
partial and -0."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(6, 6, 6), (32, 10, 7), (33, 34, 9), (34, 7, 66), (35, 12, 12), (72, 8, 6)])
def test_sweeps_match_oracle(gpu_lib, shape):
    dsg = gpu_lib
    from oracle import Oracle
    n = [m - 2 for m in shape]
    inp = dsg.config.droplet(n[0] if n[0] % 2 == 0 else n[0] + 1).replace(nx=shape[0], ny=shape[1], nz=shape[2])
    ora, gpu = Oracle(inp.as_dict()), dsg.Solver(inp)
    r = np.random.default_rng(shape[0])
    full = tuple(shape)
    cc = np.where(r.random(full) < 0.3, r.random(full), np.where(r.random(full) < 0.3, 1.0, 0.0))
    cc[r.random(full) < 0.4] = 0.0
    cc[2, 2, 2], cc[-2, -2, -2], cc[1, 1, 1] = -0.0, 1.0, 1.0
    fields = {"cc": cc}
    for k in ("u", "v", "w"):
        fields[k] = r.uniform(-1.0, 1.0, full)
    tau = 0.3 * ora.scalars().h
    for name, f in fields.items():
        f = np.asfortranarray(f)
        ora.field(name)[...] = f
        gpu.set_field(name, f)
    for x in (ora, gpu):
        s = x.scalars()
        s.tau, s.tauh = tau, 0.3
        x.set_scalars(s)
    for _ in range(3):  # the three sweep orders
        ora.vofmethod()
        gpu.vofmethod()
        a, b = gpu.field("cc"), ora.field("cc")
        assert relerr(a, b) <= 1e-12  # libm's pow, acos and cos differ by ulps
