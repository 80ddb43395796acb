"""The coarse levels in one thread-block cluster (mgcluster.cuh): the same
bits as one launch per pass (FP32) and as the oracle's mglin (FP64, exact
order), at sizes where slabs and rows end raggedly: one, two and three planes
per block, rows of odd length, fewer planes than blocks, levels that one block
runs alone, flat and tall grids, injection and trilinear prolongation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(16, 16, 16), (20, 20, 20), (24, 24, 24), (48, 48, 48), (80, 80, 80), (64, 32, 64), (32, 64, 16),
          (24, 40, 88), (96, 48, 24)]


def _grid(dsg, shape, **kw):
    base = dsg.config.droplet(shape[0], impact_speed=2.0, **kw)
    return base.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2)


@pytest.mark.parametrize("prolong", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_cluster_matches_passes(gpu_lib, shape, prolong):
    """One outer iteration of two V-cycles after the full-multigrid start, so
    that the solve's length does not depend on its convergence."""
    dsg = gpu_lib
    base = _grid(dsg, shape, mode=dsg.config.MODE_TOL_MIXED, tol=1e-9).replace(
        mg32_prolong=prolong, inner_vcycles=2, max_vcycles=2)
    out = {}
    for key, nodes in (("pass", -1), ("cluster", 0)):
        with dsg.Solver(base.replace(tail_nodes=nodes)) as s:
            try:
                s.step(1)
            except dsg.DsgError:
                pass  # two V-cycles need not reach the tolerance
            out[key] = s.field("p")
    assert np.isfinite(out["pass"]).all() and np.abs(out["pass"]).max() > 0
    assert np.array_equal(out["pass"], out["cluster"])


@pytest.mark.parametrize("shape", SHAPES[:4] + SHAPES[5:])
def test_fp64_cluster_matches_oracle(gpu_lib, shape):
    dsg = gpu_lib
    from oracle import Oracle
    inp = _grid(dsg, shape, mode=dsg.config.MODE_REF_EXACT)
    ora, gpu = Oracle(inp.as_dict()), dsg.Solver(inp)
    ora.step(1)  # a realistic right-hand side and coefficients
    for name in ("rhs", "a", "b", "c", "ei"):
        gpu.set_field(name, ora.field(name))
    s, so = gpu.scalars(), ora.scalars()
    for f in ("npre", "npost", "ntop"):
        setattr(s, f, getattr(so, f))
    gpu.set_scalars(s)
    ora.mglin()
    gpu.mglin()
    assert np.array_equal(gpu.field("p"), ora.field("p"))
