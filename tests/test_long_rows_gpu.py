"""Cooperative phases of levels with long rows (channels), where the halo and not
the cells decides the kernel's form: the bits of one launch per pass, on the
finest level and the one below it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(256, 32, 32), (320, 40, 120), (512, 64, 64), (704, 16, 64), (288, 24, 8)]


@pytest.mark.parametrize("sweeps,prolong", [(1, 1), (4, 0)])
@pytest.mark.parametrize("shape", SHAPES)
def test_long_rows_match_passes(gpu_lib, shape, sweeps, prolong):
    dsg = gpu_lib
    base = dsg.config.droplet(shape[0], impact_speed=2.0, mode=dsg.config.MODE_TOL_MIXED, tol=1e-9)
    base = base.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2, mg32_prolong=prolong, mg32_npre=sweeps,
                        mg32_npost=sweeps, inner_vcycles=2, max_vcycles=2)
    r = [(np.arange(n + 2) - 0.5) / n - 0.5 for n in shape]
    d = 0.35 - np.sqrt(r[0][:, None, None] ** 2 + r[1][None, :, None] ** 2 + r[2][None, None, :] ** 2)
    cc = np.asfortranarray(np.clip(d * min(shape) + 0.5, 0.0, 1.0))
    out = {}
    for nodes in (-1, 0):
        with dsg.Solver(base.replace(tail_nodes=nodes)) as s:
            s.set_field("cc", cc)
            try:
                s.step(1)
            except dsg.DsgError as e:  # two V-cycles need not reach the tolerance
                assert e.code == -4
            out[nodes] = s.field("p")
    assert np.isfinite(out[-1]).all() and np.abs(out[-1]).max() > 0
    assert np.array_equal(out[-1], out[0])
