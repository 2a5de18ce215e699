"""The stage kernels against the C oracle bit for bit, at the sizes where they can
go wrong.  Which kernel runs where: test_gpu_kernel_choice.py.
"""
import numpy as np
import pytest

from oracle_lib import ghost_cells, smooth_random_state

torch = pytest.importorskip("torch")

import alsvinn_b200 as als  # noqa: E402
from alsvinn_b200 import domain  # noqa: E402

pytestmark = pytest.mark.gpu


def _flux_case(c_oracle, dim, n, recon, flux, start=(0, 0, 0), end=(0, 0, 0)):
    g = ghost_cells(recon, flux)
    st = smooth_random_state(sum(n) + len(recon), dim, n, g)
    cfg = c_oracle.config(dim, n, [0.0] * dim, [1.0] * dim, flux, recon, "rungekutta3", "periodic", 1.4)
    st = c_oracle.fill_ghosts(cfg, st)
    expect, ws = c_oracle.net_flux(cfg, st)
    out = torch.full(st.shape, -7.0, dtype=torch.float64, device="cuda")
    got_ws = als.NumericalFlux(dim, n, flux, recon).computeFlux(torch.from_numpy(st).cuda(), out,
                                                                 start, end)
    box = [slice(None)]
    for d in (2, 1, 0):
        box.append(slice(g + start[d], g + n[d] + end[d]) if d < dim else slice(None))
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[tuple(box)], expect[tuple(box)])
    # nothing outside the region is written
    got[tuple(box)] = -7.0
    assert (got == -7.0).all()
    return got_ws, ws


LARGE = [(32, 12600), (12601, 33), (703, 631), (1023, 401), (1025, 399), (353, 331), (272, 265)]
RECONS = ["none", "weno2", "eno2", "eno3", "eno4", "mc", "mm", "wenof2", "weno3"]


@pytest.mark.parametrize("n", LARGE, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("recon", ["weno2", "eno4"])
def test_marching_rows_sizes(c_oracle, n, recon):
    got, ws = _flux_case(c_oracle, 2, n, recon, "hll3")
    np.testing.assert_array_equal(got[:2], ws[:2])


@pytest.mark.parametrize("recon", RECONS)
@pytest.mark.parametrize("flux", ["hll", "hll3", "central"])
def test_marching_rows_schemes(c_oracle, recon, flux):
    got, ws = _flux_case(c_oracle, 2, (801, 503), recon, flux)
    np.testing.assert_array_equal(got[:2], ws[:2])


@pytest.mark.parametrize("recon", RECONS)
def test_tiles_schemes(c_oracle, recon):
    got, ws = _flux_case(c_oracle, 2, (301, 263), recon, "hll3")
    np.testing.assert_array_equal(got[:2], ws[:2])


def test_marching_rows_regions(c_oracle):
    _flux_case(c_oracle, 2, (811, 603), "weno2", "hll3", start=(3, 2, 0), end=(-5, -1, 0))
    _flux_case(c_oracle, 2, (811, 703), "eno3", "hll", start=(0, 40, 0), end=(-70, 0, 0))


@pytest.mark.parametrize("n", [(7, 9), (16, 7), (17, 8), (33, 64), (260, 252)],
                         ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("recon", ["none", "weno2", "eno3", "weno3"])
def test_faces_2d(c_oracle, n, recon):
    got, ws = _flux_case(c_oracle, 2, n, recon, "hll3")
    np.testing.assert_array_equal(got[:2], ws[:2])


@pytest.mark.parametrize("n", [(8, 8, 8), (9, 5, 7), (17, 13, 10), (33, 40, 41), (40, 41, 42)],
                         ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("recon", ["weno2", "mc"])
def test_3d(c_oracle, n, recon):
    got, ws = _flux_case(c_oracle, 3, n, recon, "hll3")
    np.testing.assert_array_equal(got, ws)


@pytest.mark.parametrize("n", [4, 5, 127, 128, 254, 1000], ids=str)
@pytest.mark.parametrize("recon", ["none", "weno2"])
def test_faces_1d(c_oracle, n, recon):
    got, ws = _flux_case(c_oracle, 1, (n,), recon, "hll")
    np.testing.assert_array_equal(got[:1], ws[:1])


@pytest.mark.parametrize("dim,n", [(2, (700, 579)), (2, (400, 270)), (3, (33, 47, 41)), (3, (50, 16, 81))],
                         ids=["700x579", "400x270", "33x47x41", "50x16x81"])
@pytest.mark.parametrize("integ", ["rungekutta3", "rungekutta2", "forwardeuler"])
@pytest.mark.parametrize("bc", ["periodic", "neumann"])
def test_marching_steps(c_oracle, dim, n, integ, bc):
    st = smooth_random_state(5 + dim, dim, n, 2)
    cfg = c_oracle.config(dim, n, [0.0] * dim, [1.0] * dim, "hll3", "weno2", integ, bc, 1.4)
    rc, expect, dts, steps, t = c_oracle.simulate(cfg, st, 0.4, 1.0, max_steps=3)
    with als.Simulator(dim, n, flux="hll3", reconstruction="weno2", integrator=integ, boundary=bc,
                       cfl=0.4, end_time=1.0, max_steps=3) as sim:
        sim.set_state(st)
        sim.run()
        info = sim.info()
        np.testing.assert_array_equal(sim.get_state()[0], expect)
    assert info["steps"] == steps and info["t"] == t


MARCHING = [(2, (703, 632), (1, 4), "rows"), (2, (300, 280), (2, 1), "small tiles"),
            (3, (60, 48, 50), (1, 2, 2), "columns"), (3, (40, 36, 35), (2, 1, 1), "tiles")]


@pytest.mark.parametrize("dim,n,procs,kernel", MARCHING, ids=["%s-%s" % (c[3], "x".join(map(str, c[1]))) for c in MARCHING])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("bc", ["periodic", "neumann"])
def test_persistent_and_split_launches(dim, n, procs, kernel, precision, bc):
    """Persistent launches and a grid split into subdomains (ghost layers
    written across them by the stage kernels) give the bits of the plain run."""
    g = ghost_cells("weno2")
    st = smooth_random_state(11 + dim, dim, n, g)
    common = dict(flux="hll3", reconstruction="weno2", integrator="rungekutta3", boundary=bc, cfl=0.4,
                  end_time=1.0, max_steps=3, precision=precision)
    out = []
    for blocks in (0, 1):
        with als.Simulator(dim, n, **common) as sim:
            assert sim.kernels() == [kernel]
            sim.set_schedule(blocks)
            sim.set_state(st)
            sim.run()
            out.append(sim.get_state()[0])
    np.testing.assert_array_equal(out[1], out[0])
    split = domain.SplitSimulation(dim, n, procs, **common)
    try:
        assert split.sim.kernels() == [kernel]
        split.set_state(st)
        split.run()
        blocks = split.sim.get_state()
        for r, dec in enumerate(split.decs):
            np.testing.assert_array_equal(blocks[r], out[0][dec.local_slice(g)])
    finally:
        split.close()


LINES = [4, 9, 63, 64, 127, 128, 129, 255, 256, 511, 513, 1000, 2047, 4097, 8192, 8193]


@pytest.mark.parametrize("n", LINES)
@pytest.mark.parametrize("integ", ["rungekutta3", "rungekutta2"])
@pytest.mark.parametrize("bc", ["periodic", "neumann"])
def test_lines(c_oracle, n, integ, bc):
    states = np.stack([smooth_random_state(n + m, 1, (n,), 2) for m in range(3)])
    cfg = c_oracle.config(1, (n,), [0.0], [1.0], "hll3", "weno2", integ, bc, 1.4)
    end = 0.4 / n
    runs = [c_oracle.simulate(cfg, s, 0.4, end) for s in states]
    with als.Simulator(1, (n,), flux="hll3", reconstruction="weno2", integrator=integ, boundary=bc,
                       cfl=0.4, end_time=end, members=3) as sim:
        sim.set_state(states)
        sim.advance(1)          # steps split over calls
        sim.run()
        got = sim.get_state()
        for m, (rc, expect, dts, steps, t) in enumerate(runs):
            info = sim.info(m)
            assert info["steps"] == steps and info["t"] == t and info["dt"] == dts[-1]
            np.testing.assert_array_equal(got[m], expect)


@pytest.mark.parametrize("recon", RECONS)
@pytest.mark.parametrize("flux", ["hll", "hll3"])
def test_line_schemes(c_oracle, recon, flux):
    n, g = 300, ghost_cells(recon, flux)
    st = smooth_random_state(len(recon), 1, (n,), g)
    cfg = c_oracle.config(1, (n,), [0.0], [1.0], flux, recon, "rungekutta3", "neumann", 1.4)
    rc, expect, dts, steps, t = c_oracle.simulate(cfg, st, 0.4, 1.0, max_steps=4)
    with als.Simulator(1, (n,), flux=flux, reconstruction=recon, integrator="rungekutta3",
                       boundary="neumann", cfl=0.4, end_time=1.0, max_steps=4) as sim:
        sim.set_state(st)
        sim.run()
        assert sim.info()["steps"] == steps
        np.testing.assert_array_equal(sim.get_state()[0], expect)


def test_line_constraint_violation_reports_the_first_cell(c_oracle):
    n = 700
    st = smooth_random_state(1, 1, (n,), 2)
    st[-1, ..., 400:403] = 1e-3           # negative pressure
    cfg = c_oracle.config(1, (n,), [0.0], [1.0], "hll", "weno2", "rungekutta3", "periodic", 1.4)
    rc, expect, dts, steps, t = c_oracle.simulate(cfg, st, 0.4, 0.1)
    with als.Simulator(1, (n,), flux="hll", reconstruction="weno2", cfl=0.4, end_time=0.1,
                       members=2) as sim:
        good = smooth_random_state(2, 1, (n,), 2)
        sim.set_state(np.stack([good, st]))
        with pytest.raises(als._lib.AlsError):
            sim.run()
        bad, fine = sim.info(1), sim.info(0)
    assert rc != 0 and bad["status"] != 0 and bad["steps"] == steps and bad["bad_step"] == steps
    assert 380 < bad["bad_index"] < 430
    assert fine["status"] == 0 and fine["t"] == 0.1


BAD = [(1, (300,), "weno2", "hll3", 1), (2, (40, 30), "weno2", "hll3", 3), (2, (300, 270), "weno2", "hll3", 1),
       (2, (703, 631), "weno2", "hll3", 1), (2, (200, 100), "none", "tecno4", 2),
       (3, (20, 18, 16), "weno2", "hll3", 1), (3, (50, 47, 44), "weno2", "hll3", 1),
       (3, (50, 47, 44), "eno3", "hll3", 1)]


@pytest.mark.parametrize("dim,n,recon,flux,members", BAD,
                         ids=["%s-%s-%s" % ("x".join(map(str, c[1])), c[2], c[3]) for c in BAD])
def test_reported_cell_is_the_first_violation(dim, n, recon, flux, members):
    """Several cells of one thread violate the constraints (some columns, over
    all rows and planes): bad_index is the smallest padded index of them all,
    in every stage kernel."""
    g = ghost_cells(recon, flux)
    states = np.stack([smooth_random_state(17 + m, dim, n, g) for m in range(members)])
    states[:, -1, :, :, g + n[0] // 3:g + n[0] // 3 + max(3, n[0] // 3)] = 1e-3   # negative pressure
    with als.Simulator(dim, n, flux=flux, reconstruction=recon, cfl=0.4, end_time=1.0, max_steps=1,
                       members=members) as sim:
        sim.set_state(states)
        with pytest.raises(als._lib.AlsError):
            sim.run()
        for m in range(members):
            U = sim.get_state(m, 1)[0]
            with np.errstate(all="ignore"):
                p = (1.4 - 1) * (U[-1] - 0.5 * sum(U[1 + d] * U[1 + d] for d in range(dim)) / U[0])
                ok = np.isfinite(U).all(0) & (U[0] > 0) & (p > 0)
            inner = np.zeros(ok.shape, bool)
            inner[tuple(slice(g, g + n[d]) if d < dim else slice(None) for d in (2, 1, 0))] = True
            bad = np.flatnonzero(inner & ~ok)
            assert len(bad) > 1 and sim.info(m)["bad_index"] == bad[0]


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-14), ("fp32", 1e-14)])
@pytest.mark.parametrize("members", [1, 63, 64, 65, 128, 130])
def test_statistics_chunks(precision, bar, members):
    """Whole chunks of 64 states stay in registers; mean and variance against
    two-pass FP64 sums (each a sum of at most 130 terms: 130 x 2^-53)."""
    dtype = torch.float64 if precision == "fp64" else torch.float32
    g = torch.Generator().manual_seed(members)
    states = (3.0 + torch.randn(members, 4, 5, 777, generator=g, dtype=torch.float64)).to(dtype).cuda()
    mv = als.MeanVariance(states[0].numel())
    mv.add(states, precision)
    mean = torch.empty(states.shape[1:], dtype=torch.float64, device="cuda")
    var = torch.empty_like(mean)
    mv.result(mean, var)
    mv.close()
    x = states.double()
    assert float((mean - x.mean(0)).abs().max()) < 130 * bar
    assert float((var - x.var(0, unbiased=False)).abs().max()) < 130 * bar
