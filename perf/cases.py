"""The work users have this framework do, as measurable cases.

Each case is a dict of plain values.  ``prepare`` makes what a program holds
before the call (inputs on the GPU, the solver or network it keeps), ``run``
makes one pass through the public classes of ``alsvinn_b200`` and returns
whole outputs, ``exact`` restates the result in plain torch FP64.

Families ("kind"):
  sod        a whole 1-D shock-tube run from host state to host state
  solver     time steps of one grid or an ensemble of one grid size, states
             handed over on the device (2-D and 3-D, FP64 and FP32)
  levels     time steps of a multilevel ensemble and its per-level statistics
  plugin     one Runge-Kutta step through the plug-in classes
  stats      ensemble mean and variance
  structure  structure functions of an ensemble
  forward    surrogate inference
  train      surrogate training
"""
import math

import numpy as np
import torch

import alsvinn_b200 as als
from alsvinn_b200.functionals import structure_functions

GAMMA = 1.4


def listed():
    return [
        # the reference's Sod configuration, run to its end time: 498 steps of
        # 1024 cells, the latency-bound end of the range
        dict(name="sod_1024", kind="sod", n=1024, members=1, recon="weno2", flux="hll",
             integrator="rungekutta3", cfl=0.45, end=0.2),
        # a small 2-D grid, as in convergence studies and first runs
        dict(name="kh_128", kind="solver", dim=2, nx=128, ny=128, nz=1, members=1, recon="weno2",
             flux="hll3", integrator="rungekutta3", boundary="periodic", precision="fp64",
             data="kh", cfl=0.4, steps=32),
        # the Kelvin-Helmholtz headline grid, FP64 as the drop-in runs it
        dict(name="kh_1024", kind="solver", dim=2, nx=1024, ny=1024, nz=1, members=1,
             recon="weno2", flux="hll3", integrator="rungekutta3", boundary="periodic",
             precision="fp64", data="kh", cfl=0.4, steps=16),
        # another scheme on a ragged rectangle with walls: third-order ENO,
        # HLL, two stages, a few members of a developed flow
        dict(name="eno3_253x187", kind="solver", dim=2, nx=253, ny=187, nz=1, members=5,
             recon="eno3", flux="hll", integrator="rungekutta2", boundary="neumann",
             precision="fp64", data="vortices", cfl=0.4, steps=16),
        # the batched UQ ensemble with FP32 members
        dict(name="ensemble_fp32", kind="solver", dim=2, nx=256, ny=256, nz=1, members=512,
             recon="weno2", flux="hll3", integrator="rungekutta3", boundary="periodic",
             precision="fp32", data="kh", cfl=0.4, steps=8),
        # the uneven multilevel batch (a quarter of its members) with FP64 statistics
        dict(name="multilevel_fp32", kind="levels", n0=128, count=4, members0=512,
             precision="fp32", cfl=0.4, steps=8),
        # the 3-D spot check, FP64
        dict(name="kh3d_128", kind="solver", dim=3, nx=128, ny=128, nz=128, members=2,
             recon="weno2", flux="hll3", integrator="rungekutta3", boundary="periodic",
             precision="fp64", data="vortices", cfl=0.4, steps=4),
        # the reference's own loop over plug-in flux, integrator and boundary
        dict(name="plugin_512", kind="plugin", nx=512, ny=512, recon="weno2", flux="hll3",
             integrator="rungekutta3", boundary="periodic", cfl=0.4),
        # mean and variance of a quarter-thousand FP32 states, in two additions
        dict(name="stats_fp32", kind="stats", n=256, members=256, precision="fp32"),
        # cube structure functions of an ensemble snapshot
        dict(name="structure_256", kind="structure", dim=2, n=256, members=32, precision="fp32",
             mode="cube", H=8, p=1, boundary="periodic"),
        # surrogate inference for the control variate's moments
        dict(name="surrogate_forward", kind="forward", rows=1 << 20, width=256, hidden=4),
        # surrogate training at the configuration's batch
        dict(name="surrogate_train", kind="train", rows=1024, width=256, hidden=4, steps=25),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]; odd ones as likely as even."""
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["sod", "solver2", "solver2", "ensemble", "solver3", "levels", "plugin",
                       "stats", "structure", "forward", "train"])
    recon = rng.choice(["weno2", "weno2", "mc", "eno3"])
    flux = rng.choice(["hll3", "hll"])
    integrator = rng.choice(["rungekutta3", "rungekutta3", "rungekutta2"])
    boundary = rng.choice(["periodic", "neumann"])
    cfl = rng.choice([0.4, 0.45])
    if kind == "sod":
        n = _log_int(rng, 64, 3000)
        end = 0.2 * rng.uniform(0.5, 1.0) * min(1.0, 1024.0 / n)
        return dict(kind="sod", n=n, members=rng.randint(1, 6), recon=recon, flux=flux,
                    integrator=integrator, cfl=cfl, end=end)
    common = dict(recon=recon, flux=flux, integrator=integrator, cfl=cfl)
    if kind == "solver2":
        nx, ny = _log_int(rng, 24, 1100), _log_int(rng, 24, 1100)
        members = _log_int(rng, 1, max(1, min(8, (1 << 20) // (nx * ny))))
        return dict(kind="solver", dim=2, nx=nx, ny=ny, nz=1, members=members, boundary=boundary,
                    precision=rng.choice(["fp64", "fp64", "fp32"]), data="vortices",
                    steps=rng.randint(4, 16), **common)
    if kind == "ensemble":
        n = _log_int(rng, 32, 300)
        members = _log_int(rng, 8, max(8, min(2000, (1 << 23) // (n * n))))
        common["recon"] = rng.choice(["weno2", "mc"])
        return dict(kind="solver", dim=2, nx=n, ny=n, nz=1, members=members, boundary="periodic",
                    precision=rng.choice(["fp32", "fp32", "fp64"]), data=rng.choice(["kh", "vortices"]),
                    steps=rng.randint(2, 8), **common)
    if kind == "solver3":
        nx, ny, nz = (_log_int(rng, 16, 140) for _ in range(3))
        members = _log_int(rng, 1, max(1, min(4, (1 << 22) // (nx * ny * nz))))
        return dict(kind="solver", dim=3, nx=nx, ny=ny, nz=nz, members=members, boundary=boundary,
                    precision=rng.choice(["fp64", "fp64", "fp32"]), data="vortices",
                    steps=rng.randint(2, 4), **common)
    if kind == "levels":
        precision = rng.choice(["fp32", "fp64"])
        return dict(kind="levels", n0=_log_int(rng, 32, 128), count=rng.randint(2, 4),
                    members0=4 ** rng.randint(3, 4) * rng.randint(1, 2), precision=precision,
                    cfl=cfl, steps=rng.randint(2, 8) if precision == "fp32" else rng.randint(1, 3))
    if kind == "plugin":
        return dict(kind="plugin", nx=_log_int(rng, 32, 1024), ny=_log_int(rng, 32, 1024),
                    boundary=boundary, **common)
    if kind == "stats":
        return dict(kind="stats", n=_log_int(rng, 32, 256), members=_log_int(rng, 3, 300),
                    precision=rng.choice(["fp32", "fp64"]))
    if kind == "structure":
        dim = rng.choice([2, 2, 3])
        n = _log_int(rng, 32, 256) if dim == 2 else _log_int(rng, 16, 40)
        return dict(kind="structure", dim=dim, n=n, members=_log_int(rng, 1, 32 if dim == 2 else 8),
                    precision=rng.choice(["fp32", "fp64"]), mode=rng.choice(["cube", "cube", "basic"]),
                    H=rng.randint(3, 8 if dim == 2 else 5), p=rng.choice([1, 2, 3]),
                    boundary=boundary)
    if kind == "forward":
        return dict(kind="forward", rows=_log_int(rng, 100, 1 << 20), width=rng.choice([256, 256, 128]),
                    hidden=rng.randint(2, 5))
    return dict(kind="train", rows=_log_int(rng, 64, 1024), width=rng.choice([256, 256, 128]),
                hidden=rng.randint(2, 5), steps=rng.randint(5, 25))


# ---------------------------------------------------------------- inputs


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 11)
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _conserved(rho, vel, p):
    uu = sum(v * v for v in vel)
    return torch.stack([rho] + [rho * v for v in vel] + [p / (GAMMA - 1) + 0.5 * rho * uu], dim=1)


def _axes(dim, n):
    """Midpoint coordinates per direction, shaped to broadcast over (members, z, y, x)."""
    shapes = ((1, 1, 1, -1), (1, 1, -1, 1), (1, -1, 1, 1))
    return [((torch.arange(n[d], device="cuda", dtype=torch.float64) + 0.5) / n[d]).reshape(shapes[d])
            for d in range(dim)]


def _kelvin_helmholtz(g, members, dim, n):
    """Two streams with perturbed interfaces, the benchmark's initial data."""
    ax = _axes(dim, n)
    s = ax[0] if dim == 2 else ax[0] + ax[2]
    edge = []
    for base in (0.25, 0.75):
        a = _uniform(g, 0, 1, members, 10)
        a = a / a.sum(1, keepdim=True)
        b = _uniform(g, 0, 1, members, 10)
        e = torch.zeros((members,) + tuple(s.shape[1:]), device="cuda", dtype=torch.float64)
        for i in range(10):
            e += a[:, i].reshape(-1, 1, 1, 1) * torch.cos(b[:, i].reshape(-1, 1, 1, 1) +
                                                         2 * math.pi * (i + 1) * s)
        edge.append(base + 0.01 * e)
    middle = (ax[1] > edge[0]) & (ax[1] < edge[1])
    rho = torch.where(middle, 2.0, 1.0).to(torch.float64)
    ux = torch.where(middle, -0.5, 0.5).to(torch.float64)
    shape = (members,) + tuple(n[:dim][::-1]) if dim == 3 else (members, 1, n[1], n[0])
    rho, ux = rho.expand(shape), ux.expand(shape)
    zero = torch.zeros_like(rho)
    return _conserved(rho, [ux] + [zero] * (dim - 1), torch.full_like(rho, 2.5))


def _vortices(g, members, dim, n):
    """A developed flow: density, velocities and pressure vary over many
    scales, with one steep density layer."""
    ax = _axes(dim, n)

    def field():
        f = 0
        for k in range(1, 5):
            ph = _uniform(g, 0, 2 * math.pi, members, 3)
            amp = _uniform(g, 0.4, 1.0, members).reshape(-1, 1, 1, 1) / k
            term = amp
            for d in range(dim):
                term = term * torch.sin(2 * math.pi * (k + d % 2) * ax[d] + ph[:, d].reshape(-1, 1, 1, 1))
            f = f + term
        return f

    rho = 1.5 + 0.5 * torch.tanh(60.0 * (field() - 0.1)) + 0.05 * field()
    vel = [0.4 * field() for _ in range(dim)]
    p = 2.5 + 0.3 * field()
    return _conserved(rho, vel, p)


def _sod(seed, members, n):
    r = np.random.default_rng(seed * 31 + 5)
    x = -1.0 + 2.0 * (np.arange(n) + 0.5) / n
    out = np.zeros((members, 3, 1, 1, n))
    for m in range(members):
        left = x < 0
        rho = np.where(left, 1.0 + 0.05 * r.random(), 0.125 + 0.02 * r.random())
        p = np.where(left, 1.0 + 0.05 * r.random(), 0.1 + 0.02 * r.random())
        out[m, 0, 0, 0], out[m, 2, 0, 0] = rho, p / (GAMMA - 1)
    return out


def _pad(interior, dim, g):
    """Padded planes with zero ghosts (the solver fills them)."""
    pad = []
    for d in range(3):
        pad += [g, g] if d < dim else [0, 0]
    return torch.nn.functional.pad(interior, pad).contiguous()


def _dtype(precision):
    return torch.float64 if precision == "fp64" else torch.float32


def _sizes(case):
    return tuple(case[k] for k in ("nx", "ny", "nz"))[:case.get("dim", 2)]


def _upper(n):
    """Cells of equal length in every direction: the longest side has length 1."""
    return [v / max(n) for v in n]


def _states(case, seed):
    """Interior states (members, nvar, z, y, x) in the case's precision."""
    n = _sizes(case)
    make = _kelvin_helmholtz if case["data"] == "kh" else _vortices
    return make(_generator(seed), case["members"], case["dim"], n).to(_dtype(case["precision"]))


def _levels_of(case):
    out = []
    for k in range(case["count"]):
        n = case["n0"] * 2 ** k
        out.append((n, max(1, case["members0"] // 4 ** k)))
    return out


def _level_states(case, seed, k):
    n, members = _levels_of(case)[k]
    return _kelvin_helmholtz(_generator(seed * 10 + k), members, 2, (n, n)).to(_dtype(case["precision"]))


def _network(case, seed):
    """Parameters of the size a trained network has (He-scaled weights)."""
    r = np.random.default_rng(seed * 17 + 3)
    sizes = [40] + [case["width"]] * case["hidden"] + [1]
    parts = []
    for a, b in zip(sizes[:-1], sizes[1:]):
        parts.append(r.standard_normal((b, a)) * math.sqrt(2.0 / a) * (1.0 if b > 1 else 0.5))
        parts.append(r.uniform(-0.2, 0.2, b))
    return np.concatenate([p.ravel() for p in parts]).astype(np.float32)


def _samples(case, seed):
    g = _generator(seed)
    x = torch.rand(case["rows"], 40, generator=g, device="cuda", dtype=torch.float32)
    w = torch.randn(40, generator=g, device="cuda", dtype=torch.float32) / 6.0
    t = torch.tanh((x - 0.5) @ w * 3) + 0.2 * torch.randn(case["rows"], generator=g, device="cuda")
    return x, t.contiguous()


class _DeviceArray:
    """A solver's state buffer as something torch can view; the view keeps the solver alive."""

    def __init__(self, sim, like):
        self.sim = sim
        self.__cuda_array_interface__ = {
            "data": (sim.state_pointer(), False), "shape": tuple(like.shape), "version": 2,
            "typestr": "<f8" if like.dtype == torch.float64 else "<f4"}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sod":
        sim = als.Simulator(1, (case["n"],), (-1.0,), (1.0,), flux=case["flux"],
                            reconstruction=case["recon"], integrator=case["integrator"],
                            boundary="neumann", gamma=GAMMA, cfl=case["cfl"],
                            end_time=case["end"], members=case["members"])
        interior = _sod(seed, case["members"], case["n"])
        g = sim.ghosts
        host = np.zeros((case["members"],) + sim.shape)
        host[..., g:-g] = interior
        return dict(case=case, sim=sim, host=host)
    if kind == "solver":
        n = _sizes(case)
        sim = als.Simulator(case["dim"], n, None, _upper(n), flux=case["flux"],
                            reconstruction=case["recon"], integrator=case["integrator"],
                            boundary=case["boundary"], gamma=GAMMA, cfl=case["cfl"],
                            end_time=100.0, precision=case["precision"], members=case["members"])
        return dict(case=case, sim=sim, states=_pad(_states(case, seed), case["dim"], sim.ghosts))
    if kind == "levels":
        levels = [dict(n=(n, n), members=m) for n, m in _levels_of(case)]
        sim = als.Simulator(2, levels=levels, flux="hll3", reconstruction="weno2",
                            integrator="rungekutta3", boundary="periodic", gamma=GAMMA,
                            cfl=case["cfl"], end_time=100.0, precision=case["precision"])
        states = [_pad(_level_states(case, seed, k), 2, sim.ghosts) for k in range(len(levels))]
        return dict(case=case, sim=sim, states=states)
    if kind == "plugin":
        n = (case["nx"], case["ny"])
        flux = als.NumericalFlux(2, n, case["flux"], case["recon"], gamma=GAMMA)
        g = flux.getNumberOfGhostCells()
        inner = _vortices(_generator(seed), 1, 2, n)
        u0 = _pad(inner, 2, g)[0]
        integ = als.Integrator(case["integrator"], flux, case["cfl"])
        vols = [u0] + [torch.zeros_like(u0) for _ in range(integ.getNumberOfSubsteps())]
        return dict(case=case, integ=integ, boundary=als.Boundary(2, n, g, case["boundary"]),
                    vols=vols, lengths=[u / v for u, v in zip(_upper(n), n)] + [0.0])
    if kind == "stats":
        n = case["n"]
        states = _pad(_vortices(_generator(seed), case["members"], 2, (n, n)), 2, 2)
        return dict(case=case, states=states.to(_dtype(case["precision"])))
    if kind == "structure":
        n = (case["n"],) * case["dim"]
        states = _pad(_vortices(_generator(seed), case["members"], case["dim"], n), case["dim"], 2)
        return dict(case=case, states=states.to(_dtype(case["precision"])))
    net = als.Surrogate(width=case["width"], hidden=case["hidden"], max_batch=1024)
    params = _network(case, seed)
    net.set_params(params)
    x, t = _samples(case, seed)
    return dict(case=case, net=net, params=params, x=x, t=t)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sod":
        sim = state["sim"]
        sim.set_state(state["host"])
        sim.run()
        clocks = [sim.info(m) for m in range(case["members"])]
        return dict(state=sim.get_state(), t=np.array([c["t"] for c in clocks]),
                    steps=np.array([c["steps"] for c in clocks]))
    if kind == "solver":
        sim = state["sim"]
        sim.set_state_device(state["states"].data_ptr())
        sim.advance(case["steps"])
        return torch.as_tensor(_DeviceArray(sim, state["states"]), device="cuda")
    if kind == "levels":
        sim = state["sim"]
        for lev, s in zip(sim.levels, state["states"]):
            sim.set_state_device(s.data_ptr(), lev["first"], lev["members"])
        sim.advance(case["steps"])
        out = {"coarsest": torch.as_tensor(_DeviceArray(sim, state["states"][0]), device="cuda")}
        for k, lev in enumerate(sim.levels):
            mv = als.MeanVariance(4 * lev["plane"])
            mv.add_solver(sim, k)
            mean = torch.empty(lev["shape"], device="cuda", dtype=torch.float64)
            var = torch.empty_like(mean)
            mv.result(mean, var)
            mv.close()
            out["mean%d" % k], out["variance%d" % k] = mean, var
        return out
    if kind == "plugin":
        vols, integ = state["vols"], state["integ"]
        state["boundary"].applyBoundaryConditions(vols[0])
        dt = 0.0
        for s in range(integ.getNumberOfSubsteps()):
            dt = integ.performSubstep(vols, state["lengths"], dt, vols[s + 1], s, 0.0, 100.0)
            state["boundary"].applyBoundaryConditions(vols[s + 1])
        return dict(state=vols[-1], dt=dt)
    if kind == "stats":
        states = state["states"]
        half = states.shape[0] // 2
        mv = als.MeanVariance(states[0].numel())
        for part in (states[:half], states[half:]):
            if part.shape[0]:
                mv.add(part, case["precision"])
        mean = torch.empty(states.shape[1:], device="cuda", dtype=torch.float64)
        var = torch.empty_like(mean)
        mv.result(mean, var)
        mv.close()
        return dict(mean=mean, variance=var)
    if kind == "structure":
        return structure_functions(state["states"], case["dim"], (case["n"],) * case["dim"], 2,
                                   boundary=case["boundary"], kind=case["mode"], H=case["H"],
                                   p=float(case["p"]), gamma=GAMMA)
    if kind == "forward":
        return state["net"](state["x"])
    net = state["net"]
    net.set_params(state["params"])
    loss = net.train_raw(state["x"], state["t"], case["steps"], lr=1e-3)
    return dict(loss=loss, params=net.params())


# ------------------------------------------------------------ FP64 restatement


def _ghosts(case_recon):
    return {"weno2": 2, "mc": 2, "eno3": 3}[case_recon]


def _fill(U, dim, g, bc):
    """Pads interior states with their boundary images."""
    for d in range(dim):
        ax = 4 - d
        n = U.shape[ax]
        i = torch.arange(-g, n + g, device=U.device)
        if bc == "periodic":
            i = i % n
        else:
            i = torch.where(i < 0, -1 - i, torch.where(i >= n, 2 * n - 1 - i, i))
        U = U.index_select(ax, i)
    return U


def _reconstruct(U, ax, recon):
    """Left and right values of every cell but the outermost g - 1 along axis `ax`."""
    g = _ghosts(recon)
    n = U.shape[ax]

    def at(o, V=U):
        return V.narrow(ax, g - 1 + o, n - 2 * (g - 1))

    if recon == "mc":
        l, m, r = at(-1), at(0), at(1)
        a, b, c = 2 * (r - m), (r - l) / 2, 2 * (m - l)
        same = (torch.sign(a) == torch.sign(b)) & (torch.sign(b) == torch.sign(c))
        s = torch.where(same, torch.sign(a) * torch.minimum(a.abs(), torch.minimum(b.abs(), c.abs())),
                        torch.zeros((), device=U.device, dtype=U.dtype))
        return m - s / 2, m + s / 2
    rho = U[:, :1]
    if recon == "weno2":
        dp, dm = at(1, rho) - at(0, rho), at(0, rho) - at(-1, rho)
        d0, d1 = ((1e-8 + x * x) * 3 * (1e-8 + x * x) for x in (dp, dm))
        wl0, wl1 = d1 / (d1 + 2 * d0), 2 * d0 / (d1 + 2 * d0)
        wr0, wr1 = 2 * d1 / (2 * d1 + d0), d0 / (2 * d1 + d0)
        um, u0, up = at(-1), at(0), at(1)
        return (0.5 * (wl1 * um + (3 * wl0 + wl1) * u0 - wl0 * up),
                0.5 * (wr0 * up + (3 * wr1 + wr0) * u0 - wr1 * um))
    # eno3: the smoother of the neighbouring stencils, difference by difference
    d1 = rho.narrow(ax, 1, n - 1) - rho.narrow(ax, 0, n - 1)
    d2 = d1.narrow(ax, 1, n - 2) - d1.narrow(ax, 0, n - 2)

    def diff(D, o):
        return D.narrow(ax, g - 1 + o, n - 2 * (g - 1))

    shift = (diff(d1, -1).abs() < diff(d1, 0).abs()).to(torch.int64) + (
        diff(d2, -1).abs() < diff(d2, 0).abs()).to(torch.int64)
    coef = [[11 / 6, -7 / 6, 1 / 3], [1 / 3, 5 / 6, -1 / 6], [-1 / 6, 5 / 6, 1 / 3],
            [1 / 3, -7 / 6, 11 / 6]]
    left = right = None
    for s in range(3):
        lv = sum(coef[s][j] * at(j - s) for j in range(3))
        rv = sum(coef[s + 1][j] * at(j - s) for j in range(3))
        left = lv if s == 0 else torch.where(shift == s, lv, left)
        right = rv if s == 0 else torch.where(shift == s, rv, right)
    return left, right


def _primitive(U, d):
    nsd = U.shape[1] - 2
    rho = U[:, 0]
    dot = sum(U[:, 1 + k] * U[:, 1 + k] for k in range(nsd))
    p = (GAMMA - 1) * (U[:, -1] - 0.5 * dot / rho)
    return rho, U[:, 1 + d] / rho, p


def _point(U, u, p, d):
    F = U * u.unsqueeze(1)
    F[:, 0] = U[:, 1 + d]
    F[:, 1 + d] = F[:, 1 + d] + p
    F[:, -1] = (U[:, -1] + p) * u
    return F


def _face_flux(L, R, d, flux):
    rl, ul, pl = _primitive(L, d)
    rr, ur, pr = _primitive(R, d)
    wl, wr = rl.sqrt(), rr.sqrt()
    rho = (rl + rr) / 2
    u = (wl * ul + wr * ur) / (wl + wr)
    p = (wl * pl + wr * pr) / (wl + wr)
    cs = (GAMMA * p / rho).sqrt()
    cl, cr = (GAMMA * pl / rl).sqrt(), (GAMMA * pr / rr).sqrt()
    correct = 0.5 * torch.clamp(ul - ur, min=0) if flux == "hll3" else 0.0
    sL = torch.minimum(ul + correct - cl, u - cs)
    sR = torch.maximum(ur - correct + cr, u + cs)
    FL, FR = _point(L, ul, pl, d), _point(R, ur, pr, d)
    sl, sr = sL.unsqueeze(1), sR.unsqueeze(1)
    if flux == "hll":
        star = (sr * FL - sl * FR + sr * sl * (R - L)) / (sr - sl)
    else:
        dl, dr = ul - sL, ur - sR
        aa = dr * rr - dl * rl
        sm = (R[:, 1 + d] * dr - L[:, 1 + d] * dl + pr - pl) / aa
        us = [sm if k == d else (R[:, 1 + k] * ur - L[:, 1 + k] * ul - sR * R[:, 1 + k] +
                                 sL * L[:, 1 + k]) / aa for k in range(L.shape[1] - 2)]
        left = (sm >= 0).unsqueeze(1)

        def side(U, F, r, uu, pp, s, du):
            m0 = r * du / (sm - s)
            ps = pp + r * (uu - sm) * du
            e = (du * U[:, -1] + pp * uu - ps * sm) / (sm - s)
            return F + s.unsqueeze(1) * (torch.stack([m0] + [v * m0 for v in us] + [e], 1) - U)

        star = torch.where(left, side(L, FL, rl, ul, pl, sL, dl), side(R, FR, rr, ur, pr, sR, dr))
    zero = torch.zeros((), device=L.device, dtype=L.dtype)
    F = torch.where(sl == 0, zero, torch.where(sl > 0, FL, torch.where(sr < 0, FR, star)))
    return F, torch.maximum(sL.abs(), sR.abs())


def _net_flux(U, dim, recon, flux, bc):
    """Net flux of interior states U and the largest face speeds (members, dim)."""
    g = _ghosts(recon)
    out, speeds = torch.zeros_like(U), []
    full = _fill(U, dim, g, bc)
    for d in range(dim):
        V = full
        for e in range(dim):
            if e != d:
                V = V.narrow(4 - e, g, U.shape[4 - e])
        ax = 4 - d
        l, r = _reconstruct(V, ax, recon)
        faces = U.shape[ax] + 1
        F, w = _face_flux(r.narrow(ax, 0, faces), l.narrow(ax, 1, faces), d, flux)
        out = out + (F.narrow(ax, 0, faces - 1) - F.narrow(ax, 1, faces - 1))
        speeds.append(w.flatten(1).amax(1))
    return out, torch.stack(speeds, 1)


def _march(U, dim, n, case, bc, steps=None, end=100.0, lengths=None):
    """Whole time steps of interior FP64 states; returns (U, t, steps) per member."""
    recon, flux = case.get("recon", "weno2"), case.get("flux", "hll3")
    rk3 = case.get("integrator", "rungekutta3") == "rungekutta3"
    dx = torch.tensor(lengths, device=U.device, dtype=torch.float64)
    M = U.shape[0]
    t = torch.zeros(M, device=U.device, dtype=torch.float64)
    count = torch.zeros(M, device=U.device, dtype=torch.int64)
    k = 0
    while steps is None or k < steps:
        if steps is None and k % 8 == 0 and bool((t >= end).all()):
            break
        L, ws = _net_flux(U, dim, recon, flux, bc)
        live = t < end
        dt = torch.minimum(case["cfl"] / (ws / dx).sum(1), end - t)
        c = (dt / dx[0]).reshape(-1, 1, 1, 1, 1)
        U1 = L * c + U
        if rk3:
            U2 = ((_net_flux(U1, dim, recon, flux, bc)[0] * c + U1) * (1 / 3) + U) * (3 / 4)
            V = ((_net_flux(U2, dim, recon, flux, bc)[0] * c + U2) * 2 + U) * (1 / 3)
        else:
            V = ((_net_flux(U1, dim, recon, flux, bc)[0] * c + U1) + U) * 0.5
        U = torch.where(live.reshape(-1, 1, 1, 1, 1), V, U)
        t = torch.where(live, t + dt, t)
        count += live
        k += 1
    return U, t, count


def _march_chunks(U, *args, **kwargs):
    """_march over blocks of members, to bound the temporaries."""
    per = max(1, (1 << 24) // U[0].numel())
    return torch.cat([_march(U[a:a + per].double(), *args, **kwargs)[0]
                      for a in range(0, U.shape[0], per)])


def _mlp(case, params, x):
    """Output of the network in FP64 (GELU in its tanh form)."""
    sizes = [40] + [case["width"]] * case["hidden"] + [1]
    at, h = 0, x
    for k, (a, b) in enumerate(zip(sizes[:-1], sizes[1:])):
        W = params[at:at + a * b].reshape(b, a)
        bias = params[at + a * b:at + a * b + b]
        at += a * b + b
        h = h @ W.T + bias
        if k < len(sizes) - 2:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    return h[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "sod":
        n, g = case["n"], _ghosts(case["recon"])
        U = torch.from_numpy(_sod(seed, case["members"], n)).cuda()
        U, t, steps = _march(U, 1, (n,), case, "neumann", None, case["end"], [2.0 / n])
        return dict(state=_fill(U, 1, g, "neumann"), t=t, steps=steps)
    if kind == "solver":
        n = _sizes(case)
        lengths = [u / v for u, v in zip(_upper(n), n)]
        U = _march_chunks(_states(case, seed), case["dim"], n, case, case["boundary"], case["steps"],
                          lengths=lengths)
        return _fill(U, case["dim"], _ghosts(case["recon"]), case["boundary"])
    if kind == "levels":
        out = {}
        for k, (n, _) in enumerate(_levels_of(case)):
            U = _march_chunks(_level_states(case, seed, k), 2, (n, n), case, "periodic",
                              case["steps"], lengths=[1.0 / n] * 2)
            U = _fill(U, 2, 2, "periodic")
            if k == 0:
                out["coarsest"] = U
            out["mean%d" % k] = U.mean(0)
            out["variance%d" % k] = U.var(0, unbiased=False)
        return out
    if kind == "plugin":
        n = (case["nx"], case["ny"])
        lengths = [u / v for u, v in zip(_upper(n), n)]
        U = _vortices(_generator(seed), 1, 2, n)
        V, t, _ = _march(U, 2, n, case, case["boundary"], 1, lengths=lengths)
        return dict(state=_fill(V, 2, _ghosts(case["recon"]), case["boundary"])[0], dt=float(t[0]))
    if kind == "stats":
        n = case["n"]
        states = _pad(_vortices(_generator(seed), case["members"], 2, (n, n)), 2, 2)
        states = states.to(_dtype(case["precision"])).double()
        return dict(mean=states.mean(0), variance=states.var(0, unbiased=False))
    if kind == "structure":
        dim, H, p = case["dim"], case["H"], case["p"]
        n = (case["n"],) * dim
        U = _vortices(_generator(seed), case["members"], dim, n)
        U = U.to(_dtype(case["precision"])).double()
        big = U.clone()
        for d in range(dim):
            i = torch.arange(-H, n[d] + H, device=U.device)
            i = i % n[d] if case["boundary"] == "periodic" else i.clamp(0, n[d] - 1)
            big = big.index_select(4 - d, i)
        out = torch.zeros(U.shape[0], U.shape[1], H, device=U.device, dtype=torch.float64)

        def add(h, off):
            V = big
            for d in range(dim):
                V = V.narrow(4 - d, H + off[d], n[d])
            out[:, :, h] += (U - V).abs().pow(p).flatten(2).sum(2)

        for h in range(1, H):
            if case["mode"] == "basic":
                add(h, (h, 0, 0))
                continue
            span = range(-h, h + 1)
            for ox in span:
                for oy in span:
                    for oz in (span if dim == 3 else (0,)):
                        if max(abs(ox), abs(oy), abs(oz)) == h:
                            add(h, (ox, oy, oz))
        return out / U[0, 0].numel()
    params = torch.from_numpy(_network(case, seed)).cuda().double()
    x, t = _samples(case, seed)
    if kind == "forward":
        return torch.cat([_mlp(case, params, part.double()) for part in x.split(1 << 18)])
    x, t = x.double(), t.double()
    params.requires_grad_(True)
    m, v = torch.zeros_like(params), torch.zeros_like(params)
    losses = []
    for k in range(1, case["steps"] + 1):
        loss = (_mlp(case, params, x) - t).square().mean()
        (grad,) = torch.autograd.grad(loss, params)
        losses.append(loss.detach())
        with torch.no_grad():
            m.mul_(0.9).add_(grad, alpha=0.1)
            v.mul_(0.999).addcmul_(grad, grad, value=0.001)
            params -= 1e-3 * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return dict(loss=torch.stack(losses), params=params.detach())


# ------------------------------------------------------------ work, tolerance


def _solver_work(cells, nv, dim, steps, stages, elem, recon):
    """A step's CFL reduction needs the whole state, so every step reads and
    writes it; the arithmetic counts each +, *, / and sqrt of the method once."""
    per_recon = {"weno2": 24 + 12 * nv, "mc": 14 * nv, "eno3": 8 + 22 * nv}[recon]
    per_face = 90 + 14 * dim
    per_cell = dim * (per_recon + per_face + 3 * nv) + 6 * nv
    return {"bytes": 2.0 * cells * nv * elem * steps, "flops": float(cells) * per_cell * steps * stages}


def work(case):
    kind = case["kind"]
    stages = 3 if case.get("integrator", "rungekutta3") == "rungekutta3" else 2
    elem = 8 if case.get("precision", "fp64") == "fp64" else 4
    if kind == "sod":
        steps = max(1, int(498 * case["end"] / 0.2 * case["n"] / 1024 * 0.45 / case["cfl"]))
        return _solver_work(case["n"] * case["members"], 3, 1, steps, stages, 8, case["recon"])
    if kind == "solver":
        cells = case["members"] * math.prod(_sizes(case))
        return _solver_work(cells, case["dim"] + 2, case["dim"], case["steps"], stages, elem,
                            case["recon"])
    if kind == "levels":
        cells = sum(n * n * m for n, m in _levels_of(case))
        w = _solver_work(cells, 4, 2, case["steps"], 3, elem, "weno2")
        w["bytes"] += sum(2 * 8.0 * 4 * n * n for n, _ in _levels_of(case))
        return w
    if kind == "plugin":
        return _solver_work(case["nx"] * case["ny"], 4, 2, 1, stages, 8, case["recon"])
    if kind == "stats":
        count = 4 * (case["n"] + 4) ** 2
        return {"bytes": float(count) * (case["members"] * elem + 16), "flops": 5.0 * count * case["members"]}
    if kind == "structure":
        values = case["members"] * (case["dim"] + 2) * float(case["n"] ** case["dim"])
        if case["mode"] == "basic":
            points = case["H"] - 1
        elif case["dim"] == 2:
            points = sum(8 * h for h in range(1, case["H"]))
        else:
            points = sum(24 * h * h + 2 for h in range(1, case["H"]))
        return {"bytes": values * elem, "flops": values * points * (2 + case["p"])}
    weights = 40 * case["width"] + (case["hidden"] - 1) * case["width"] ** 2 + case["width"]
    if kind == "forward":
        return {"bytes": case["rows"] * 41 * 4.0 + weights * 4, "flops": 2.0 * case["rows"] * weights}
    return {"bytes": case["steps"] * weights * 4 * 6.0 + case["rows"] * 41 * 4,
            "flops": 6.0 * case["steps"] * case["rows"] * weights}


def tolerance(case):
    """About four times the measured distance from exact() (FP32 and BF16
    paths); FP64 simulations are reproducible to the bit."""
    kind = case["kind"]
    fp64 = case.get("precision", "fp64") == "fp64"
    if kind in ("sod", "plugin"):
        return "exact"
    if kind == "solver":
        return "exact" if fp64 else {"rel": 5e-6}
    if kind == "levels":
        # the variance of nearly equal members amplifies FP32 rounding
        return {"rel": 1e-12} if fp64 else {"rel": 3e-5}
    if kind in ("stats", "structure"):
        return {"rel": 1e-12}
    if kind == "forward":
        return {"rel": 4e-2}
    return {"rel": 8e-3}
