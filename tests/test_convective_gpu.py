"""k_convective shares its two-point sums between neighbouring cells: a step's
velocities against the oracle where the tiles are ragged -- rows of 2 and of 34
cells beyond a warp's 32, rows that do not fill a block, 2 to 16 planes per
block with a remainder."""
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-10


@pytest.mark.parametrize("shape", [(34, 20, 28), (66, 12, 36), (96, 44, 140), (68, 100, 300)])
def test_step_velocities(gpu_lib, shape):
    dsg = gpu_lib
    from oracle import Oracle
    inp = dsg.config.droplet(shape[0], impact_speed=2.0)
    inp = inp.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2)
    ora, gpu = Oracle(inp.as_dict()), dsg.Solver(inp)
    for t in (1, 2):
        ora.step(t)
        gpu.step(t)
        for name in ("u", "v", "w"):
            assert relerr(gpu.field(name), ora.field(name)) <= FIELD_TOL, (t, name)
