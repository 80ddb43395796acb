"""V-cycles without sweeps on the way down or up: the fixed-cycle FP64 solve
gives the oracle's bits and the FP32 levels those of one launch per pass, at
sizes whose levels run as cooperative phases where they have sweeps (registers,
mggrid.cuh, and shared memory, mgbox.cuh)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SWEEPS = [(0, 2), (0, 0), (2, 0), (-1, 1)]


def _grid(dsg, shape, **kw):
    base = dsg.config.droplet(shape[0], impact_speed=2.0, **kw)
    return base.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2)


@pytest.mark.parametrize("npre,npost", SWEEPS)
@pytest.mark.parametrize("shape", [(48, 48, 48), (72, 76, 80), (96, 40, 52)])
def test_fp64_matches_oracle(gpu_lib, shape, npre, npost):
    dsg = gpu_lib
    from oracle import Oracle
    inp = _grid(dsg, shape, mode=dsg.config.MODE_REF_EXACT)
    ora = Oracle(inp.as_dict())
    ora.step(1)  # a realistic right-hand side and coefficients
    with dsg.Solver(inp) as gpu:
        for name in ("rhs", "a", "b", "c", "ei"):
            gpu.set_field(name, ora.field(name))
        s, so = gpu.scalars(), ora.scalars()
        so.npre, so.npost = npre, npost
        ora.set_scalars(so)
        for f in ("npre", "npost", "ntop"):
            setattr(s, f, getattr(so, f))
        gpu.set_scalars(s)
        ora.mglin()
        for _ in range(5):
            gpu.mglin()
            assert np.array_equal(gpu.field("p"), ora.field("p"))


@pytest.mark.parametrize("prolong", [0, 1])
@pytest.mark.parametrize("npre,npost", SWEEPS)
@pytest.mark.parametrize("shape", [(66, 34, 50), (72, 76, 84), (192, 192, 192)])
def test_fp32_matches_passes(gpu_lib, shape, npre, npost, prolong):
    """mg32_npre and mg32_npost of 0 leave the sweeps to the scalars."""
    dsg = gpu_lib
    base = _grid(dsg, shape, mode=dsg.config.MODE_TOL_MIXED, tol=1e-9).replace(
        mg32_prolong=prolong, mg32_npre=0, mg32_npost=0, mg32_fine_npre=0, mg32_fine_npost=0, mg32_mid_npre=0,
        mg32_mid_npost=0, mg32_small_npre=0, mg32_small_npost=0, inner_vcycles=2, max_vcycles=2)
    out = {}
    for key, nodes in (("pass", -1), ("phase", 0)):
        with dsg.Solver(base.replace(tail_nodes=nodes)) as s:
            x = s.scalars()
            x.npre, x.npost = npre, npost
            s.set_scalars(x)
            try:
                s.step(1)
            except dsg.DsgError:
                pass  # two V-cycles need not reach the tolerance
            out[key] = s.field("p")
    assert np.abs(out["pass"]).max() > 0
    assert np.array_equal(out["pass"], out["phase"], equal_nan=True)
