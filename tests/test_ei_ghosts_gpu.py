"""The ghosts of ei after a whole step: zero beyond the upper faces, where bc_flux
puts zeros in each VOF sweep, and untouched elsewhere, as in the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 16, 16), (34, 20, 12)])
@pytest.mark.parametrize("mode", [0, 2])
def test_ei_ghosts_match_oracle(gpu_lib, shape, mode):
    dsg = gpu_lib
    from oracle import Oracle
    inp = dsg.config.droplet(shape[0], impact_speed=2.0, tol=1e-8)
    inp = inp.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2)
    ora, gpu = Oracle(inp.as_dict()), dsg.Solver(inp.replace(mode=mode))
    ei = np.asfortranarray(np.random.default_rng(1).random(ora.shape))
    ora.field("ei")[...] = ei
    gpu.set_field("ei", ei)
    ora.step(1)
    try:
        gpu.step(1)
    except dsg.DsgError as e:  # the long grid's solve stops at its cycle cap; the step is complete
        assert e.code == -4
    ghost = np.ones(ora.shape, bool)
    ghost[1:-1, 1:-1, 1:-1] = False
    a, b = gpu.field("ei")[ghost], ora.field("ei")[ghost]
    assert np.array_equal(a, b)
    assert np.count_nonzero(b == 0.0) > 0
    gpu.close()
