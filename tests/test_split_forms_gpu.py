"""The finest FP32 level's forms for cells in one fluid -- four cells of a sweep,
one or two coarse cells of a restriction per thread -- against the general one:
with 1e-30 in place of 0 the volume fractions are no longer uniform, but no
coefficient changes in any precision, so the solve must give the same bits.
Sides where the rows end inside a segment, a pair of coarse cells and a block,
below and above the sizes from which the forms are used."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prolong", [0, 1])
@pytest.mark.parametrize("shape", [(64, 48, 40), (88, 80, 72), (136, 152, 168), (200, 144, 120), (264, 112, 128)])
def test_uniform_forms_match_general(gpu_lib, shape, prolong):
    dsg = gpu_lib
    inp = dsg.config.droplet(shape[0], impact_speed=2.0, mode=dsg.config.MODE_TOL_MIXED, tol=1e-9).replace(
        nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2, mg32_prolong=prolong, inner_vcycles=2, max_vcycles=2,
        tail_nodes=-1)
    with dsg.Solver(inp) as s:
        try:
            s.step(1)  # coefficients and a right-hand side
        except dsg.DsgError:
            pass  # two V-cycles need not reach the tolerance
        cc, rhs = s.field("cc"), s.field("rhs")
        rhs = np.random.default_rng(1).standard_normal(rhs.shape) * max(float(np.abs(rhs).max()), 1.0)
        out = []
        for value in (0.0, 1e-30):
            s.set_field("cc", np.where(cc == 0.0, value, cc))
            s.set_field("rhs", rhs)
            s.set_field("p", np.zeros_like(rhs))
            try:
                s.mglin()
            except dsg.DsgError:
                pass
            out.append(s.field("p"))
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1])
