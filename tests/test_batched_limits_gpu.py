"""Which members a batched solve takes: those whose coarsest level has at most
18^3 nodes, or tail_nodes, whatever their own solves run in a cluster."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(dsg, side, nodes):
    return [dsg.config.droplet(n, mode=dsg.config.MODE_TOL_MIXED, tol=1e-4, impact_speed=2.0, seed=n).replace(
        tail_nodes=nodes) for n in (32, side)]


# coarsest levels of 19^3 and 25^3 cells, and of 2^3 (4^3 = 64 nodes) below tail_nodes
@pytest.mark.parametrize("side,nodes", [(38, 0), (50, 0), (32, 63), (32, -1)])
def test_refused(gpu_lib, side, nodes):
    dsg = gpu_lib
    with dsg.Ensemble(_inputs(dsg, side, nodes), workers=2) as e:
        with pytest.raises(dsg.DsgError) as ex:
            e.set_batched(1)
        assert ex.value.code == -1 and "coarse tail is off" in str(ex.value)


@pytest.mark.parametrize("side,nodes", [(48, 0), (38, 10000)])
def test_accepted(gpu_lib, side, nodes):
    dsg = gpu_lib
    inputs = _inputs(dsg, side, nodes)
    alone = []
    for inp in inputs:
        with dsg.Solver(inp) as s:
            s.step(1)
            alone.append(s.field("p"))
    with dsg.Ensemble(inputs, workers=2, batched=1) as e:
        e.step(1)
        for i, p in enumerate(alone):
            assert np.array_equal(e.member(i).field("p"), p), i
