"""The finest FP32 sweep's uniform segments (mg32_cells.cuh): steps on grids
whose rows end inside a segment and inside a warp, against the FP64 tolerance
mode, which does not use them (sides that coarsen to a few cells, so that the
FP64 multigrid converges).  Both solves reach 1e-10; a wrong coefficient
anywhere would keep the mixed solve from converging or change its pressure."""
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(80, 80, 80), (96, 96, 48), (160, 80, 80), (160, 160, 80)])
def test_steps_match_fp64(gpu_lib, shape):
    dsg = gpu_lib
    assert (shape[0] // 2) % 4 == 0 and shape[0] // 2 * shape[1] * shape[2] >= 200000
    inp = dsg.config.droplet(shape[0], impact_speed=2.0, tol=1e-10).replace(
        nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2)
    out = {}
    for mode in (dsg.config.MODE_TOL_FP64, dsg.config.MODE_TOL_MIXED):
        with dsg.Solver(inp.replace(mode=mode)) as s:
            for t in (1, 2):
                st = s.step(t)
                assert st["converged"] == 1
            out[mode] = {f: s.field(f) for f in ("p", "u", "v", "w", "cc")}
    for f in ("p", "u", "v", "w", "cc"):
        assert relerr(out[dsg.config.MODE_TOL_MIXED][f], out[dsg.config.MODE_TOL_FP64][f]) < 1e-7, f
