"""Two solvers stepped by two host threads at once, each on its own stream: their
cluster launches and cooperative phases meet on the GPU, and each gives the bits
it gives alone, in the FP64 modes and the mixed one, with and without graphs."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 6


def _run(dsg, inp, start, out, key):
    try:
        with dsg.Solver(inp) as s:
            start.wait(60)
            for t in range(1, STEPS + 1):
                s.step(t)
            out[key] = {f: s.field(f) for f in ("p", "u", "v", "w", "cc")}
    except Exception as e:  # reported by the main thread
        out[key] = e


@pytest.mark.parametrize("a,b", [((64, 0, 1), (48, 0, 1)), ((64, 2, 1), (96, 2, 1)), ((80, 2, 0), (64, 1, 1)),
                                 ((192, 2, 1), (48, 2, 1))])
def test_two_threads(gpu_lib, a, b):
    dsg = gpu_lib
    inputs = [dsg.config.droplet(n, impact_speed=2.0, mode=m, tol=1e-8, seed=n).replace(use_graphs=g)
              for n, m, g in (a, b)]
    alone, both = {}, {}
    for k, inp in enumerate(inputs):
        _run(dsg, inp, threading.Barrier(1), alone, k)
    start = threading.Barrier(2)
    ts = [threading.Thread(target=_run, args=(dsg, inp, start, both, k)) for k, inp in enumerate(inputs)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k in range(2):
        assert isinstance(alone[k], dict) and isinstance(both[k], dict), (alone[k], both[k])
        for f in alone[k]:
            assert np.array_equal(alone[k][f], both[k][f]), (k, f)
