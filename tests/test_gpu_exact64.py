"""The straight-line FP64 division and root of the HLL / HLL3 fluxes and the
WENO2 weights (csrc/exact64.cuh, euler_exact64.cuh) against the C oracle, bit
for bit: states inside their tested ranges, on both sides of the ranges'
edges, and the mantissas the rounding proofs single out.  The oracle divides
with the host's IEEE operators, so the expected difference is zero.
"""
import numpy as np
import pytest

from oracle_lib import ghost_cells, padded_shape

torch = pytest.importorskip("torch")

import alsvinn_b200 as als  # noqa: E402

pytestmark = pytest.mark.gpu

GAMMA = 1.4
SIZES = {1: (300,), 2: (40, 37), 3: (18, 17, 9)}


def _ordinary(dim, rng, shape):
    """Conserved states with rough densities, velocities and pressures."""
    rho = rng.uniform(0.2, 3.0, shape[1:])
    vel = rng.uniform(-1.5, 1.5, (dim,) + shape[1:])
    p = rng.uniform(0.1, 3.0, shape[1:])
    E = p / (GAMMA - 1) + 0.5 * rho * (vel * vel).sum(0)
    return np.concatenate([rho[None], rho * vel, E[None]])


def _states(kind, dim, rng, shape):
    U = _ordinary(dim, rng, shape)
    if kind == "ordinary":
        return U
    if kind == "supersonic":
        U[1:1 + dim] *= 8.0
        U[-1] += 32.0 * U[0]
    elif kind == "signed_zero":
        U[1:1 + dim] = np.where(rng.random(U[1:1 + dim].shape) < 0.5, 0.0, -0.0)
        U[0] = np.where(rng.random(shape[1:]) < 0.5, 1.0, 2.0)
        U[-1] = 6.25
    elif kind == "tiny_momentum":
        # across 2^-700 and into the subnormals
        e = rng.integers(-1074, -600, U[1:1 + dim].shape)
        m = np.ldexp(rng.uniform(1, 2, e.shape), e.astype(np.int32))
        U[1:1 + dim] = np.where(rng.random(e.shape) < 0.3, 0.0, m) * rng.choice([-1, 1], e.shape)
        U[-1] = rng.uniform(1, 4, shape[1:])
    elif kind == "range_edges":
        # densities and energies across 2^-60 and 2^60
        s = np.ldexp(1.0, rng.choice([-64, -61, -60, -59, 58, 59, 60, 62, 120], shape[1:]).astype(np.int32))
        U = U * s
    elif kind == "mantissas":
        # all ones, 1 + last place, powers of two: the hard cases of 1/d and sqrt
        ones = 2.0 - 2.0 ** -52
        pick = np.array([ones, 1.0 + 2.0 ** -52, 1.0, ones * 2, ones * 0.5, 2.0 + 2.0 ** -51])
        U[0] = rng.choice(pick, shape[1:])
        U[1:1 + dim] = rng.choice(pick, U[1:1 + dim].shape) * rng.choice([-1, 1], U[1:1 + dim].shape)
        U[-1] = rng.choice(pick, shape[1:]) * 64
    elif kind == "unphysical":
        # negative densities and pressures, infinities and NaNs here and there
        U[0] = np.where(rng.random(shape[1:]) < 0.05, -U[0], U[0])
        U[-1] = np.where(rng.random(shape[1:]) < 0.05, 1e-3, U[-1])
        U[-1] = np.where(rng.random(shape[1:]) < 0.01, np.inf, U[-1])
        U[1] = np.where(rng.random(shape[1:]) < 0.01, np.nan, U[1])
        U[0] = np.where(rng.random(shape[1:]) < 0.01, 0.0, U[0])
    return U


KINDS = ["ordinary", "supersonic", "signed_zero", "tiny_momentum", "range_edges", "mantissas",
         "unphysical"]


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("flux", ["hll", "hll3"])
@pytest.mark.parametrize("recon", ["none", "weno2", "wenof2"])
@pytest.mark.parametrize("kind", KINDS)
def test_net_flux_equals_the_oracle(c_oracle, dim, flux, recon, kind):
    n = SIZES[dim]
    g = ghost_cells(recon)
    rng = np.random.default_rng(KINDS.index(kind) * 100 + dim * 10 + len(recon))
    st = _states(kind, dim, rng, padded_shape(dim, n, g))
    cfg = c_oracle.config(dim, n, [0.0] * dim, [1.0] * dim, flux, recon, "rungekutta3", "periodic",
                          GAMMA)
    with np.errstate(all="ignore"):
        st = c_oracle.fill_ghosts(cfg, st)
        expect, ws = c_oracle.net_flux(cfg, st)
    dev = torch.from_numpy(st).cuda()
    out = torch.zeros_like(dev)
    got_ws = als.NumericalFlux(dim, n, flux, recon, gamma=GAMMA).computeFlux(dev, out)
    got = out.cpu().numpy()
    inner = (slice(None),) + tuple(slice(g, -g) if d < dim else slice(None) for d in (2, 1, 0))
    np.testing.assert_array_equal(got[inner], expect[inner])
    # zeros keep their sign
    zero = expect[inner] == 0
    np.testing.assert_array_equal(np.signbit(got[inner][zero]), np.signbit(expect[inner][zero]))
    np.testing.assert_array_equal(got_ws[:dim], ws[:dim])


@pytest.mark.parametrize("gamma", [1.0 + 2.0 ** -30, 1.1, 5.0 / 3.0, 3000.0])
def test_adiabatic_exponents(c_oracle, gamma):
    n, g = (40, 37), 2
    rng = np.random.default_rng(3)
    st = _states("ordinary", 2, rng, padded_shape(2, n, g))
    cfg = c_oracle.config(2, n, [0.0] * 2, [1.0] * 2, "hll3", "weno2", "rungekutta3", "periodic", gamma)
    st = c_oracle.fill_ghosts(cfg, st)
    with np.errstate(all="ignore"):
        expect, ws = c_oracle.net_flux(cfg, st)
    dev = torch.from_numpy(st).cuda()
    out = torch.zeros_like(dev)
    got_ws = als.NumericalFlux(2, n, "hll3", "weno2", gamma=gamma).computeFlux(dev, out)
    np.testing.assert_array_equal(out.cpu().numpy()[:, :, g:-g, g:-g], expect[:, :, g:-g, g:-g])
    np.testing.assert_array_equal(got_ws[:2], ws[:2])


@pytest.mark.parametrize("dim,n", [(2, (301, 263)), (2, (801, 503)), (3, (40, 36, 35)), (3, (50, 47, 44)), (1, (80000,))],
                         ids=["small tiles", "rows", "boxes", "columns", "1-D tiles"])
@pytest.mark.parametrize("flux", ["hll", "hll3"])
@pytest.mark.parametrize("kind", KINDS)
def test_every_kernel_falls_back(c_oracle, dim, n, flux, kind):
    """The same states through the kernels of larger grids (their sizes above)."""
    g = 2
    rng = np.random.default_rng(KINDS.index(kind) + dim)
    st = _states(kind, dim, rng, padded_shape(dim, n, g))
    cfg = c_oracle.config(dim, n, [0.0] * dim, [1.0] * dim, flux, "weno2", "rungekutta3", "periodic",
                          GAMMA)
    with np.errstate(all="ignore"):
        st = c_oracle.fill_ghosts(cfg, st)
        expect, ws = c_oracle.net_flux(cfg, st)
    dev = torch.from_numpy(st).cuda()
    out = torch.zeros_like(dev)
    got_ws = als.NumericalFlux(dim, n, flux, "weno2", gamma=GAMMA).computeFlux(dev, out)
    inner = (slice(None),) + tuple(slice(g, -g) if d < dim else slice(None) for d in (2, 1, 0))
    np.testing.assert_array_equal(out.cpu().numpy()[inner], expect[inner])
    np.testing.assert_array_equal(got_ws[:dim], ws[:dim])


@pytest.mark.parametrize("flux", ["hll", "hll3"])
@pytest.mark.parametrize("kind", ["ordinary", "supersonic", "signed_zero", "tiny_momentum", "mantissas"])
def test_line_steps_fall_back(c_oracle, flux, kind):
    """Whole steps of a line in one launch."""
    n = 900
    st = _states(kind, 1, np.random.default_rng(9), padded_shape(1, (n,), 2))
    cfg = c_oracle.config(1, (n,), [0.0], [1.0], flux, "weno2", "rungekutta3", "periodic", GAMMA)
    with np.errstate(all="ignore"):
        rc, expect, dts, steps, t = c_oracle.simulate(cfg, c_oracle.fill_ghosts(cfg, st), 0.4, 1e300,
                                                      max_steps=1)
    with als.Simulator(1, (n,), flux=flux, reconstruction="weno2", cfl=0.4, end_time=1e300, max_steps=1) as sim:
        assert sim.kernels() == ["lines"]
        sim.set_state(st)
        sim.advance(1)
        np.testing.assert_array_equal(sim.get_state()[0], expect)
        assert sim.info()["t"] == t
