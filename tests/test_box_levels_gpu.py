"""Levels below the finest whose phases keep u and the right-hand side in shared
memory (mgbox.cuh): the bits of one launch per pass, on flat and long grids and
with boxes of different sizes, rows of 3 to 51 items, a closed interface across
most boxes, injection and trilinear prolongation, and sweep counts of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(400, 96, 208), (208, 176, 184), (144, 240, 172), (48, 360, 400), (176, 152, 200), (816, 16, 400)]


def _input(dsg, shape, **kw):
    # half the finest level's sides: beyond what the SMs' registers hold (eight
    # cells per thread and colour on 152 SMs), rows of whole items
    assert shape[0] * shape[1] * shape[2] // 8 > 152 * 256 * 16 and shape[0] % 16 == 0
    base = dsg.config.droplet(shape[0], impact_speed=2.0, mode=dsg.config.MODE_TOL_MIXED, tol=1e-9)
    return base.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2, inner_vcycles=2, max_vcycles=2, **kw)


def _ellipsoid(shape):
    r = [(np.arange(n + 2) - 0.5) / n - 0.5 for n in shape]
    d = 0.3 - np.sqrt(r[0][:, None, None] ** 2 + r[1][None, :, None] ** 2 + r[2][None, None, :] ** 2)
    return np.asfortranarray(np.clip(d * min(shape) + 0.5, 0.0, 1.0))


def _solve(dsg, inp, cc):
    with dsg.Solver(inp) as s:
        s.set_field("cc", cc)
        n0 = s.lib.dsg_launch_count()
        try:
            s.step(1)
        except dsg.DsgError as e:  # two V-cycles need not reach the tolerance
            assert e.code == -4
        return s.field("p"), s.lib.dsg_launch_count() - n0


@pytest.mark.parametrize("npre,npost,prolong", [(8, 8, 0), (1, 3, 1)])
@pytest.mark.parametrize("shape", SHAPES)
def test_box_matches_passes(gpu_lib, shape, npre, npost, prolong):
    dsg = gpu_lib
    inp = _input(dsg, shape, mg32_prolong=prolong, mg32_mid_npre=npre, mg32_mid_npost=npost)
    cc = _ellipsoid(shape)
    a, _ = _solve(dsg, inp.replace(tail_nodes=-1), cc)
    b, _ = _solve(dsg, inp.replace(tail_nodes=0), cc)
    assert np.isfinite(a).all() and np.abs(a).max() > 0
    assert np.array_equal(a, b)


@pytest.mark.parametrize("shape", SHAPES)
def test_route(gpu_lib, shape):
    """The level below the finest takes one launch per phase, however many sweeps."""
    dsg = gpu_lib
    cc = _ellipsoid(shape)
    n = {}
    for nodes in (-1, 0):
        for m in (2, 5):
            inp = _input(dsg, shape, mg32_mid_npre=m, mg32_mid_npost=m, use_graphs=0, tail_nodes=nodes)
            n[nodes, m] = _solve(dsg, inp, cc)[1]
    assert n[0, 2] == n[0, 5] and n[-1, 2] < n[-1, 5]
