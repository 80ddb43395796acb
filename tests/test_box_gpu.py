"""Smoothing phases of large levels in one cooperative launch (mgbox.cuh): the
same bits as one launch per pass, on the finest level and below it, with the
right-hand side in shared memory and not, whole and ragged boxes, both fluids
and their interface, injection and trilinear prolongation, no sweeps on the way
down."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(96, 96, 96), (128, 112, 100), (160, 160, 160), (144, 76, 200), (256, 36, 184), (192, 192, 192),
          (256, 160, 224)]


@pytest.mark.parametrize("npre,prolong", [(8, 1), (3, 0), (0, 1)])
@pytest.mark.parametrize("shape", SHAPES)
def test_box_matches_passes(gpu_lib, shape, npre, prolong):
    dsg = gpu_lib
    base = dsg.config.droplet(shape[0], impact_speed=2.0, mode=dsg.config.MODE_TOL_MIXED, tol=1e-9)
    base = base.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2, mg32_prolong=prolong, mg32_npre=npre,
                        mg32_fine_npre=min(npre, 3), inner_vcycles=2, max_vcycles=2)
    out = {}
    for key, nodes in (("pass", -1), ("box", 0)):
        with dsg.Solver(base.replace(tail_nodes=nodes)) as s:
            try:
                s.step(1)
            except dsg.DsgError:
                pass  # two V-cycles need not reach the tolerance
            out[key] = s.field("p")
    assert np.isfinite(out["pass"]).all() and np.abs(out["pass"]).max() > 0
    assert np.array_equal(out["pass"], out["box"])
