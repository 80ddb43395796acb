"""The live profile's bytes of the finest FP32 sweep: four words per cell where
uniform segments need no volume fraction, six on the grids without them."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("n,words", [(48, 6), (50, 6), (96, 4)])
def test_bytes_per_call(gpu_lib, n, words, graphs):
    dsg = gpu_lib
    inp = dsg.config.droplet(n, impact_speed=2.0, mode=dsg.config.MODE_TOL_MIXED, tol=1e-4).replace(use_graphs=graphs)
    with dsg.Solver(inp) as s:
        s.profile_enable(True)
        s.step(1)
        p = s.profile_read()
    assert p["relax_calls"] > 0 and p["relax_bits"] == 32
    assert p["relax_bytes"] == pytest.approx(p["relax_calls"] * words * 4.0 * (n + 2) ** 3)
