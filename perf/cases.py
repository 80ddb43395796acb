"""The work that users of this package have it do, as timed cases.

A case is one call sequence through the public entry points: a time step of a
simulation resident on the GPU, a time step whose state lives in the host's
arrays, one step of an ensemble, a two-grid cycle or a set of single kernels
on a host program's own device arrays, or a training pass of the network.
"""
import importlib
import math

import numpy as np
import torch

dsg = importlib.import_module("3d_droplet_simulation_2007_gb300")

MODES = dsg.config.MODE_NAMES
# A run of a small simulation goes on for this many steps, then the next run
# starts from the stored initial state (the 64^3 study case runs 200 steps).
RUN_STEPS = 200
# The state that carries from one step to the next.
STATE = ("cc", "u", "v", "w", "s12", "s13", "s23", "res", "rhs", "p")
# The state a host that owns its fields sends and takes back (bench.py's
# end-to-end step).
HOST_IN = ("cc", "u", "v", "w", "s12", "s13", "s23")
HOST_OUT = ("p", "cc", "u", "v", "w")


def _step(name, n, mode, tol, speed, npre, ny=0, nz=0, surfacet=2, hswitch=0):
    return {"name": name, "kind": "step", "n": n, "ny": ny or n, "nz": nz or n, "mode": mode, "tol": tol,
            "speed": speed, "npre": npre, "surfacet": surfacet, "hswitch": hswitch}


def listed():
    return [
        # The smallest calls: a host program's own multigrid on its device
        # arrays, one two-grid cycle over the array-level kernels at 34^3 nodes.
        {"name": "twogrid_32", "kind": "twogrid", "nx": 32, "ny": 32, "nz": 32},
        # The single kernels on a large, odd, non-cubic grid (no side coarsens).
        {"name": "arrays_ragged", "kind": "arrays", "nx": 201, "ny": 143, "nz": 173},
        # The small study configuration: the reference's fixed-cycle FP64 method.
        _step("step_ref_64", 64, "ref_exact", 1e-10, 1.0, 5),
        # The parity configuration: the same method at 128^3.
        _step("step_ref_128", 128, "ref_exact", 1e-10, 1.0, 5),
        # The reference's default surface tension (SGIP with interface heights)
        # on a side that is not a power of two, on a flat domain.
        _step("step_sgip_96", 96, "ref_exact", 1e-10, 3.0, 5, ny=48, surfacet=5, hswitch=1),
        # The splash with the plain FP64 method run to a tolerance.
        _step("step_fp64_256", 256, "tol_fp64", 1e-8, 3.0, 4),
        # The droplet study's smallest and largest members, one at a time.
        _step("step_mixed_48", 48, "tol_mixed", 1e-8, 2.0, 4),
        _step("step_mixed_160", 160, "tol_mixed", 1e-8, 4.0, 4),
        # The splash on the wall at 256^3, the headline workload.
        _step("step_mixed_256", 256, "tol_mixed", 1e-8, 3.0, 4),
        # A Fortran host that keeps its COMMON blocks: state in and out each step.
        {"name": "host_mixed_128", "kind": "host", "n": 128, "mode": "tol_mixed", "tol": 1e-8, "speed": 3.0},
        # Eight members of the droplet study stepped together.
        {"name": "ensemble_8", "kind": "ensemble", "members": 8, "largest": 128, "first": 1000},
        # A training pass of the learned start's network: forward, loss, gradient.
        {"name": "net_64", "kind": "net", "W": 64, "H": 64, "D": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "twogrid", "arrays", "host", "ensemble", "net"])
    if kind == "step":
        mode = rng.choice(["ref_exact", "tol_fp64", "tol_mixed", "tol_mixed"])
        n = rng.choice([20, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256])
        if mode != "tol_mixed":
            n = min(n, 192)
        flat = n >= 48 and n % 32 == 0 and rng.random() < 0.4
        sgip = mode == "ref_exact" and rng.random() < 0.5
        c = _step("", n, mode, rng.choice([1e-8, 1e-9, 1e-10]) if mode != "tol_mixed" else rng.choice([1e-8, 1e-9]),
                  round(rng.uniform(1.0, 5.0), 3), rng.choice([4, 5]), ny=n // 2 if flat else n,
                  nz=n // 2 if flat and rng.random() < 0.5 else n, surfacet=rng.choice([5, 6]) if sgip else 2,
                  hswitch=1 if sgip else 0)
    elif kind == "twogrid":
        c = {"kind": kind, **{a: 2 * _log_int(rng, 6, 96) for a in ("nx", "ny", "nz")}}
    elif kind == "arrays":
        c = {"kind": kind, **{a: _log_int(rng, 9, 220) for a in ("nx", "ny", "nz")}}
    elif kind == "host":
        c = {"kind": kind, "n": rng.choice([32, 48, 64, 80, 96, 128, 160]), "mode": rng.choice(["tol_mixed", "ref_exact"]),
             "tol": 1e-8, "speed": round(rng.uniform(1.0, 4.0), 3)}
    elif kind == "ensemble":
        c = {"kind": kind, "members": rng.randrange(2, 11), "largest": rng.choice([64, 96, 128]),
             "first": rng.randrange(1000, 2000)}
    else:
        c = {"kind": kind, **{a: 8 * rng.randrange(2, 11) for a in ("W", "H", "D")}}
    c.pop("name", None)
    return c


# ---- inputs ------------------------------------------------------------------

class _DeviceArray:
    """A context's field for a torch tensor over the same memory, which keeps
    the context's owner alive as long as it lives."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _view(solver, name, owner=None):
    nx, ny, nz = solver.shape
    return torch.as_tensor(_DeviceArray(solver.field_ptr(name), nx * ny * nz, owner or solver), device="cuda")


def _input(c, seed):
    inp = dsg.config.droplet(c["n"], impact_speed=c["speed"], mode=MODES[c["mode"]], tol=c["tol"],
                             npre=c.get("npre", 4), npost=c.get("npre", 4), seed=seed)
    return inp.replace(ny=c.get("ny", c["n"]) + 2, nz=c.get("nz", c["n"]) + 2, surfacet=c.get("surfacet", 2),
                       hswitch=c.get("hswitch", 0))


def _drop(shape, gen):
    """Volume fraction of a droplet at a random place: a sharp interface a few
    cells wide, 0 and 1 elsewhere (ghosts included)."""
    nz, ny, nx = shape
    ax = [torch.arange(m, dtype=torch.float64, device="cuda") - 0.5 for m in (nz, ny, nx)]
    m = min(shape) - 2
    c = [float(torch.rand((), generator=gen, device="cuda", dtype=torch.float64)) * 0.3 + 0.35 for _ in range(3)]
    r = 0.25 * m
    dist = torch.sqrt((ax[0] - c[0] * (nz - 2)).square()[:, None, None] + (ax[1] - c[1] * (ny - 2)).square()[None, :, None]
                      + (ax[2] - c[2] * (nx - 2)).square()[None, None, :])
    return torch.clamp(0.5 + (r - dist), 0.0, 1.0).contiguous()


def _arrays(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    shape = (c["nz"] + 2, c["ny"] + 2, c["nx"] + 2)

    def field(scale):
        x = torch.zeros(shape, dtype=torch.float64, device="cuda")
        x[1:-1, 1:-1, 1:-1] = scale * torch.randn([m - 2 for m in shape], generator=gen, device="cuda", dtype=torch.float64)
        return x
    s = {"cc": _drop(shape, gen), "u": field(1.0), "rhs": field(50.0)}
    for k in ("a", "b", "c", "ei", "res", "cf"):
        s[k] = torch.zeros(shape, dtype=torch.float64, device="cuda")
    if c["kind"] == "twogrid":
        coarse = tuple((m - 2) // 2 + 2 for m in shape)
        for k in ("uc", "rhsc", "ac", "bc", "cc2", "eic"):
            s[k] = torch.zeros(coarse, dtype=torch.float64, device="cuda")
    return s


R2 = 0.0012
R1 = 0.5 * (1.0 - R2)
OMEGA = 1.5
SWEEPS = 4


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = c = dict(case)
    kind = c["kind"]
    if kind == "step":
        s.solver = dsg.Solver(_input(c, seed))
        s.first = {k: s.solver.field(k) for k in STATE} if s.solver.shape[0] < 130 else None
        s.scalars = s.solver.scalars()
        s.out = {k: _view(s.solver, k) for k in ("p", "u", "v", "w", "cc")}
    elif kind == "host":
        s.solver = dsg.Solver(_input(c, seed))
        s.solver.step()  # a state in mid-flight: the first step starts the stresses
        s.scalars = s.solver.scalars()
        s.t = s.solver.t + 1
        n = int(np.prod(s.solver.shape))
        pin = {k: torch.empty(n, dtype=torch.float64, pin_memory=True) for k in HOST_IN}
        s.inputs = {k: s.solver.download_into(k, v.numpy()) for k, v in pin.items()}
        s.outputs = {k: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() for k in HOST_OUT}
    elif kind == "ensemble":
        sides = [m for m in (48, 64, 96, 128, 160) if m <= c["largest"]]
        s.ens = dsg.Ensemble(dsg.study_configs(c["members"], sides=sides, seed=c["first"]), workers=c["members"])
        for i in range(c["members"]):  # the members' noise differs with the seed, their sizes do not
            m = s.ens.member(i)
            r = np.random.default_rng([seed, i])
            for k in ("u", "v", "w"):
                f = m.field(k)
                m.set_field(k, f + 1e-4 * r.uniform(-1.0, 1.0, f.shape))
        s.out = [{k: _view(s.ens.member(i), k, s.ens) for k in ("p", "u", "v", "w", "cc")} for i in range(c["members"])]
    elif kind == "net":
        learned = importlib.import_module(dsg.__name__ + ".learned")
        s.net = learned.Net(c["W"], c["H"], c["D"], seed=seed)
        r = np.random.default_rng(seed)
        s.x = r.standard_normal((c["D"], c["H"], c["W"], 5), dtype=np.float32)
        s.target = 0.1 * r.standard_normal((c["D"], c["H"], c["W"]), dtype=np.float32)
    else:
        s.f = _arrays(c, seed)
    return s


def _restart(s):
    for k, v in s.first.items():
        s.solver.set_field(k, v)
    s.solver.set_scalars(s.scalars)
    s.solver.t = 0


def run(s):
    kind = s.case["kind"]
    if kind == "step":
        if s.first is not None and s.solver.t >= RUN_STEPS:
            _restart(s)
        s.solver.step()
        return s.out
    if kind == "host":
        s.solver.set_scalars(s.scalars)
        s.solver.step_host(s.inputs, s.outputs, s.t)
        return s.outputs
    if kind == "ensemble":
        s.ens.step()
        return s.out
    if kind == "net":
        y = s.net.forward(s.x)
        loss, g = s.net.loss_grad(s.x, s.target)
        return {"y": y, "loss": loss, "grad": g}
    K, f = dsg.kernels, s.f
    shape = tuple(reversed(f["u"].shape))
    K.abcei(f["a"], f["b"], f["c"], f["ei"], f["cc"], R1, R2, shape)
    for _ in range(SWEEPS):
        K.relax(f["u"], 1.0, f["rhs"], f["a"], f["b"], f["c"], f["ei"], shape, OMEGA)
    K.resid(1.0, f["res"], f["u"], f["rhs"], f["a"], f["b"], f["c"], shape)
    if kind == "arrays":
        K.filterc27(f["cc"], f["cf"], shape)
        K.bc("bc_out", f["cf"], shape)
        return {k: f[k] for k in ("u", "res", "a", "b", "c", "ei", "cf")}
    coarse = tuple(reversed(f["uc"].shape))
    K.rstrct(f["rhsc"], f["res"], coarse)
    K.acfromac(f["ac"], f["bc"], f["cc2"], f["eic"], f["a"], f["b"], f["c"], coarse)
    f["uc"].zero_()
    for _ in range(SWEEPS):
        K.relax(f["uc"], 1.0, f["rhsc"], f["ac"], f["bc"], f["cc2"], f["eic"], coarse, OMEGA)
    K.addint(f["u"], f["uc"], f["res"], shape)
    for _ in range(SWEEPS):
        K.relax(f["u"], 1.0, f["rhs"], f["a"], f["b"], f["c"], f["ei"], shape, OMEGA)
    return {k: f[k] for k in ("u", "uc", "res", "a", "b", "c", "ei", "rhsc", "ac", "bc", "cc2", "eic")}


# ---- least work ---------------------------------------------------------------

def _step_work(nx, ny, nz, npre):
    nodes = (nx + 2) * (ny + 2) * (nz + 2)
    cells = nx * ny * nz
    # in: cc, u, v, w, S12, S13, S23; out: those, p, S11, S22, S33, rho, mu
    words = 7 + 13
    # stress 18, predictor 20, convection 51, divergence 6, projection 6,
    # sweeps of one V-cycle and its smaller grids (17 per cell and sweep, 8/7)
    cycles = 2
    flops = cells * (101 + cycles * 2 * npre * 17 * 8 / 7)
    return {"bytes": 8.0 * words * nodes, "flops": float(flops)}


def work(case):
    c = case
    if c["kind"] == "step":
        return _step_work(c["n"], c["ny"], c["nz"], c["npre"])
    if c["kind"] == "host":
        return _step_work(c["n"], c["n"], c["n"], 4)
    if c["kind"] == "ensemble":
        sides = [m for m in (48, 64, 96, 128, 160) if m <= c["largest"]]
        each = [_step_work(x.nx - 2, x.ny - 2, x.nz - 2, 4)
                for x in dsg.study_configs(c["members"], sides=sides, seed=c["first"])]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if c["kind"] == "net":
        vox = c["W"] * c["H"] * c["D"]
        # multiply-adds of the seven layers per voxel of the finest grid
        mac = 27 * (5 * 16 + 16 * 32 / 8 + 32 * 64 / 64 + 64 * 64 / 512 + 64 * 32 / 64 + 32 * 16 / 8 + 16)
        return {"bytes": float(vox * 4 * (2 * 5 + 1 + 1) + 4 * 3 * 251649), "flops": float(2 * mac * vox * 4)}
    nodes = (c["nx"] + 2) * (c["ny"] + 2) * (c["nz"] + 2)
    cells = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "arrays":
        # in: cc, u, rhs; out: u, res, a, b, c, ei, cf
        return {"bytes": 8.0 * 10 * nodes, "flops": float(cells * (20 + SWEEPS * 17 + 19 + 30))}
    return {"bytes": 8.0 * 9 * nodes + 8.0 * 6 * nodes / 8,
            "flops": float(cells * (20 + 2 * SWEEPS * 17 + 19 + 3 + SWEEPS * 17 / 8))}


# ---- the same in plain torch, 64 bits ------------------------------------------

def _colour(shape):
    nz, ny, nx = shape
    i = torch.arange(nx, device="cuda")
    return (i[None, None, :] + torch.arange(ny, device="cuda")[None, :, None]
            + torch.arange(nz, device="cuda")[:, None, None] + 3)[1:-1, 1:-1, 1:-1] % 2


def _bc_scalar(u):
    u[:, :, 0] = u[:, :, 1]
    u[:, :, -1] = 0.0
    u[:, 0, :] = u[:, 1, :]
    u[:, -1, :] = u[:, -2, :]
    u[0] = u[1]
    u[-1] = u[-2]


IN = (slice(1, -1),) * 3


def _six(x, a, b, c, diff):
    """Sum over the six faces of coefficient times neighbour (or difference)."""
    o = x[IN] if diff else 0.0
    m, s, p = slice(1, -1), slice(0, -2), slice(2, None)
    return (a[m, m, m] * (x[m, m, p] - o) + a[m, m, s] * (x[m, m, s] - o) + b[m, m, m] * (x[m, p, m] - o)
            + b[m, s, m] * (x[m, s, m] - o) + c[m, m, m] * (x[p, m, m] - o) + c[s, m, m] * (x[s, m, m] - o))


def _relax(u, rhs, a, b, c, ei, n):
    h = 1.0 / (u.shape[2] - 2)
    col = _colour(u.shape)
    for _ in range(n):
        for q in (0, 1):
            _bc_scalar(u)
            new = OMEGA * (_six(u, a, b, c, False) - h * h * rhs[IN]) * ei[IN] + (1.0 - OMEGA) * u[IN]
            u[IN] = torch.where(col == q, new, u[IN])
    _bc_scalar(u)


def _resid(res, u, rhs, a, b, c):
    h = 1.0 / (u.shape[2] - 2)
    res[IN] = rhs[IN] - _six(u, a, b, c, True) / (h * h)
    res[:, :, 0], res[:, :, -1] = res[:, :, 1].clone(), res[:, :, -2].clone()
    res[1:-1, 0, 1:-1] = res[1:-1, -1, 1:-1] = 0.0
    res[0, :, 1:-1] = res[-1, :, 1:-1] = 0.0


def _face(cc, d):
    n = cc.shape[d] - 1
    return 1.0 / (R1 * (cc.narrow(d, 0, n) + cc.narrow(d, 1, n)) + R2)


def _sum_ei(a, b, c):
    m, s = slice(1, -1), slice(0, -2)
    return 1.0 / (a[m, m, m] + a[m, m, s] + b[m, m, m] + b[m, s, m] + c[m, m, m] + c[s, m, m])


def _exact_arrays(case, seed):
    f = _arrays(case, seed)
    m = slice(1, -1)
    cc, a, b, c, ei = f["cc"], f["a"], f["b"], f["c"], f["ei"]
    a[IN] = _face(cc, 2)[m, m, 1:]
    a[:, :, 0], a[:, :, -1] = a[:, :, 1].clone(), a[:, :, -2].clone()
    b[m, 0:-1, m] = _face(cc, 1)[m, :, m]
    c[1:-1, m, m] = _face(cc, 0)[1:, m, m]
    c[0, :, m] = _face(cc, 0)[0, :, m]
    ei[IN] = _sum_ei(a, b, c)
    _relax(f["u"], f["rhs"], a, b, c, ei, SWEEPS)
    _resid(f["res"], f["u"], f["rhs"], a, b, c)
    if case["kind"] == "arrays":
        w = [float(np.float32(x)) for x in (0.2729, 0.08185, 0.0178, 0.0028)]
        nz, ny, nx = cc.shape
        cf = torch.zeros_like(cc)
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    cf[IN] += w[abs(dz) + abs(dy) + abs(dx)] * cc[1 + dz:nz - 1 + dz, 1 + dy:ny - 1 + dy, 1 + dx:nx - 1 + dx]
        cf.clamp_(max=1.0)
        cf[:, :, 0], cf[:, :, -1] = cf[:, :, 1].clone(), cf[:, :, -2].clone()
        cf[m, 0, :], cf[m, -1, :] = cf[m, 1, :].clone(), cf[m, -2, :].clone()
        cf[0, :, m], cf[-1, :, m] = cf[1, :, m].clone(), cf[-2, :, m].clone()
        f["cf"] = cf
        return {k: f[k] for k in ("u", "res", "a", "b", "c", "ei", "cf")}

    def mean8(x):
        nz, ny, nx = x.shape
        return x.reshape(nz // 2, 2, ny // 2, 2, nx // 2, 2).mean(dim=(1, 3, 5))
    f["rhsc"][IN] = mean8(f["res"][IN])
    _bc_scalar(f["rhsc"])
    ac, bc, c2 = f["ac"], f["bc"], f["cc2"]

    def mean4(x, d):  # faces 1, 3, 5 .. along d (1-based), averaged over the 2x2 fine faces
        x = x.index_select(d, torch.arange(0, x.shape[d], 2, device="cuda"))
        for e in {0, 1, 2} - {d}:
            k = x.shape[e] - 2
            x = 0.5 * (x.narrow(e, 1, k).index_select(e, torch.arange(0, k, 2, device="cuda"))
                       + x.narrow(e, 1, k).index_select(e, torch.arange(1, k, 2, device="cuda")))
        return x
    ac[m, m, :-1], bc[m, :-1, m], c2[:-1, m, m] = mean4(a, 2), mean4(b, 1), mean4(c, 0)
    f["eic"][IN] = _sum_ei(ac, bc, c2)
    _relax(f["uc"], f["rhsc"], ac, bc, c2, f["eic"], SWEEPS)
    res = f["res"]
    up = f["uc"][IN]
    for d in (0, 1, 2):
        up = up.repeat_interleave(2, dim=d)
    res[IN] = up
    _bc_scalar(res)
    f["u"] += res
    _relax(f["u"], f["rhs"], a, b, c, ei, SWEEPS)
    return {k: f[k] for k in ("u", "uc", "res", "a", "b", "c", "ei", "rhsc", "ac", "bc", "cc2", "eic")}


def _conv(x, w, b):
    """3x3x3 convolution, zero padding, channels last; w [27][cin][cout]."""
    D, H, W, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = b
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        y = y + xp[dz:dz + D, dy:dy + H, dx:dx + W] @ w[t]
    return y


def _exact_net(case, seed):
    s = prepare(case, seed)
    layers = [(5, 16), (16, 32), (32, 64), (64, 64), (64, 32), (32, 16), (16, 1)]
    flat = torch.from_numpy(s.net.params).double().cuda().requires_grad_(True)
    x = torch.from_numpy(s.x).double().cuda()
    t = torch.from_numpy(s.target).double().cuda()
    P, at = [], 0
    for ci, co in layers:
        P.append((flat[at:at + 27 * ci * co].reshape(27, ci, co), flat[at + 27 * ci * co:at + 27 * ci * co + co]))
        at += 27 * ci * co + co

    def pool(z):
        D, H, W, C = z.shape
        return z.reshape(D // 2, 2, H // 2, 2, W // 2, 2, C).mean(dim=(1, 3, 5))

    def up(z):
        for d in (0, 1, 2):
            z = z.repeat_interleave(2, dim=d)
        return z
    e1 = _conv(x, *P[0]).relu()
    e2 = _conv(pool(e1), *P[1]).relu()
    e3 = _conv(pool(e2), *P[2]).relu()
    e4 = _conv(pool(e3), *P[3]).relu()
    d3 = _conv(up(e4) + e3, *P[4]).relu()
    d2 = _conv(up(d3) + e2, *P[5]).relu()
    y = _conv(up(d2) + e1, *P[6])[..., 0]
    loss = (y - t).square().mean()
    loss.backward()
    return {"y": y.detach(), "loss": float(loss), "grad": flat.grad}


def exact(case, seed):
    """The outputs of run() in plain 64-bit torch; none for whole steps."""
    if case["kind"] in ("twogrid", "arrays"):
        return _exact_arrays(case, seed)
    if case["kind"] == "net":
        return _exact_net(case, seed)
    return None
