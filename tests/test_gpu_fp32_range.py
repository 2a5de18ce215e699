"""FP32 members over the whole range of FP32: the hardware reciprocals and
roots that flush subnormal numbers are used only where a face's operands and
results are normal (csrc/euler_math.cuh, flush_applies), and the WENO2 weights
are scaled so that they always are.  Grids on both sides of the size rules, so
every stage kernel meets them.
"""
import numpy as np
import pytest

from oracle_lib import ghost_cells

torch = pytest.importorskip("torch")

import alsvinn_b200 as als  # noqa: E402

pytestmark = pytest.mark.gpu

GAMMA = 1.4
GRIDS = [(1, (200,)), (2, (48, 40)), (2, (300, 270)), (2, (703, 631)), (3, (18, 17, 16)), (3, (50, 47, 44)),
         (3, (65, 49, 50))]
IDS = ["x".join(map(str, n)) for _, n in GRIDS]


def _state(dim, n, g, rho, vel, p, seed=3):
    """Rough conserved states of the scales (rho, vel, p), rounded to FP32."""
    rng = np.random.default_rng(seed)
    shape = tuple(n[d] + 2 * g if d < dim else 1 for d in (2, 1, 0))
    r = rho * rng.uniform(0.9, 1.6, shape)
    u = [vel * rng.uniform(-1.5, 1.5, shape) for _ in range(dim)]
    e = p * rng.uniform(0.9, 1.6, shape) / (GAMMA - 1) + 0.5 * r * sum(v * v for v in u)
    return np.stack([r] + [r * v for v in u] + [e]).astype(np.float32).astype(np.float64)


def _run(dim, n, flux, recon, precision, st, steps):
    with als.Simulator(dim, n, flux=flux, reconstruction=recon, boundary="periodic", gamma=GAMMA,
                       cfl=0.4, end_time=1e300, precision=precision) as sim:
        sim.set_state(st)
        sim.advance(steps)
        return sim.get_state()[0], sim.info()


def _compare(dim, n, flux, recon, st, steps, tol):
    a, ia = _run(dim, n, flux, recon, "fp64", st, steps)
    b, ib = _run(dim, n, flux, recon, "fp32", st, steps)
    assert ia["status"] == 0 and ib["status"] == 0 and ib["steps"] == steps
    assert abs(ib["t"] - ia["t"]) <= tol * ia["t"]
    for v in range(dim + 2):
        scale = np.sqrt(np.mean(a[v] ** 2))
        assert np.sqrt(np.mean((a[v] - b[v]) ** 2)) <= tol * scale, v


# An FP32 value carries 2^-24; a stage's reconstruction, flux and update take
# some 30 roundings each and the flux differences cancel by up to dt/dx, so a
# few steps stay within 1e3 x 2^-24 of the FP64 run of the same state.
TOL = 1e3 * 2.0 ** -24


@pytest.mark.parametrize("dim,n", GRIDS, ids=IDS)
@pytest.mark.parametrize("recon", ["weno2", "wenof2"])
@pytest.mark.parametrize("flux", ["hll3", "hll", "central"])
@pytest.mark.parametrize("rho", [1e9, 4e9, 1e12])
def test_dense_states(dim, n, recon, flux, rho):
    """Densities whose WENO2 smoothness terms reach 2^126 and beyond."""
    _compare(dim, n, flux, recon, _state(dim, n, ghost_cells(recon), rho, 0.1, rho), 2, TOL)


@pytest.mark.parametrize("dim,n", GRIDS, ids=IDS)
@pytest.mark.parametrize("recon", ["none", "mc"])
@pytest.mark.parametrize("flux", ["hll3", "hll", "central"])
def test_reciprocal_of_the_density_below_the_normal_numbers(dim, n, recon, flux):
    """1/rho is subnormal above 2^126 = 8.5e37 (RK3 forms 3 rho, so rho stays below
    1.1e38); momenta and pressures are ordinary."""
    _compare(dim, n, flux, recon, _state(dim, n, ghost_cells(recon), 6e37, 1e-20, 1.0), 2, TOL)


@pytest.mark.parametrize("dim,n", GRIDS, ids=IDS)
@pytest.mark.parametrize("flux", ["hll3", "hll", "central"])
def test_cold_gas_keeps_its_sound_speed(dim, n, flux):
    """A gas at rest with p/rho below the normal numbers: the time step comes
    from the sound speed 1e-19 and not from zero."""
    st = _state(dim, n, ghost_cells("none"), 1.0, 0.0, 3e-39)
    a = _run(dim, n, flux, "none", "fp64", st, 1)[1]
    b = _run(dim, n, flux, "none", "fp32", st, 1)[1]
    # p has 2^-149 / 3e-39 = 5e-7 of its own
    assert abs(b["dt"] - a["dt"]) <= 1e-5 * a["dt"]


@pytest.mark.parametrize("dim,n", GRIDS, ids=IDS)
@pytest.mark.parametrize("flux", ["hll3", "hll", "central"])
def test_thin_gas(dim, n, flux):
    """Densities below the normal numbers, whose reciprocal is finite above 2^-128."""
    st = _state(dim, n, ghost_cells("none"), 6e-39, 0.0, 6e-39)
    a = _run(dim, n, flux, "none", "fp64", st, 1)[1]
    b = _run(dim, n, flux, "none", "fp32", st, 1)[1]
    assert abs(b["dt"] - a["dt"]) <= 1e-5 * a["dt"]
