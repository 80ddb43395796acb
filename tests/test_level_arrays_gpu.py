"""dsg_level_ptr: pressure, residual and right-hand side of the levels below the
finest, ghosts included, are the oracle's after a solve, on levels that a
cluster holds, on cooperative phases and on levels run pass by pass, whether
the pointers were taken before the solve or after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("p", "res", "rhs")


class _Array:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _pointers(gpu, ng):
    return {(f, l): gpu.level_ptr(f, l) for f in FIELDS for l in range(1, ng)}


def _read(torch, gpu, ptr, dims):
    gpu.synchronize()
    return torch.as_tensor(_Array(ptr, dims[0] * dims[1] * dims[2]), device="cuda").cpu().numpy().reshape(dims, order="F")


def _pair(dsg, shape, **kw):
    from oracle import Oracle
    inp = dsg.config.droplet(shape[0], impact_speed=2.0, mode=kw.pop("mode", dsg.config.MODE_REF_EXACT))
    inp = inp.replace(nx=shape[0] + 2, ny=shape[1] + 2, nz=shape[2] + 2, **kw)
    ora = Oracle(inp.as_dict())
    ora.step(1)  # a realistic right-hand side and coefficients
    gpu = dsg.Solver(inp)
    for name in ("rhs", "a", "b", "c", "ei"):
        gpu.set_field(name, ora.field(name))
    return ora, gpu


def _sweeps(ora, gpu, npre, npost):
    s, so = gpu.scalars(), ora.scalars()
    so.npre, so.npost = npre, npost
    ora.set_scalars(so)
    for f in ("npre", "npost", "ntop"):
        setattr(s, f, getattr(so, f))
    gpu.set_scalars(s)


# 128 x 96 x 64: the level below the finest is too large for a phase
@pytest.mark.parametrize("shape", [(16, 16, 16), (48, 48, 48), (40, 24, 72), (128, 96, 64)])
@pytest.mark.parametrize("cycles,npre,npost", [(2, 4, 4), (1, 0, 2), (1, 2, 0), (0, 4, 4)])
def test_levels_match_oracle(gpu_lib, shape, cycles, npre, npost):
    import torch
    dsg = gpu_lib
    ora, gpu = _pair(dsg, shape, cycles=cycles)
    ng = gpu.scalars().ng
    _sweeps(ora, gpu, npre, npost)
    ora.mglin()
    gpu.mglin()
    s = gpu.scalars()
    s.npre, s.npost, s.ntop = npre + 3, npost + 3, s.ntop + 3  # as the step's adaptivity does after a solve
    gpu.set_scalars(s)
    ptr = _pointers(gpu, ng)
    assert ng >= 2 and len(ptr) == 3 * (ng - 1)
    for (f, l), (p, dims) in ptr.items():
        assert np.array_equal(_read(torch, gpu, p, dims), ora.level_field(f, l)), (f, l)
    # the pointers stay good for the next solve
    _sweeps(ora, gpu, npre + 1, npost + 1)
    ora.mglin()
    gpu.mglin()
    for (f, l), (p, dims) in ptr.items():
        assert np.array_equal(_read(torch, gpu, p, dims), ora.level_field(f, l)), (f, l)
    gpu.close()


@pytest.mark.parametrize("shape", [(32, 32, 32), (48, 40, 56)])
def test_levels_match_oracle_to_tolerance(gpu_lib, shape):
    import torch
    dsg = gpu_lib
    ora, gpu = _pair(dsg, shape, mode=dsg.config.MODE_TOL_FP64, tol=1e-8, fp64_exact=1)
    ng = gpu.scalars().ng
    ptr = _pointers(gpu, ng)
    _sweeps(ora, gpu, 4, 4)
    ora.mglin()
    stats = gpu.mglin()
    assert stats["vcycles"] == ora.scalars().last_vcycles and stats["vcycles"] > 0
    for (f, l), (p, dims) in ptr.items():
        assert np.array_equal(_read(torch, gpu, p, dims), ora.level_field(f, l)), (f, l)
    gpu.close()
