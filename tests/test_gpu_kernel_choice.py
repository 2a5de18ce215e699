"""The rules that choose a stage kernel by size and scheme: which kernel runs on
both sides of each line, and what the launch accounting, the profile and the
tuner say of 1-D lines.  (That all kernels give the same bits:
test_gpu_batch_bits.py, test_gpu_stage_kernels.py, test_gpu_ensemble.py.)
"""
import numpy as np
import pytest

from oracle_lib import smooth_random_state

torch = pytest.importorskip("torch")

import alsvinn_b200 as als  # noqa: E402

pytestmark = pytest.mark.gpu

# dimension, n, members, reconstruction, flux, precision -> kernel
CHOICES = [
    (2, (256, 256), 1, "weno2", "hll3", "fp64", "faces"),            # 592 boxes, two rounds
    (2, (257, 256), 1, "weno2", "hll3", "fp64", "small tiles"),
    (2, (32, 32), 59, "eno4", "hll3", "fp64", "faces"),              # 590 boxes
    (2, (32, 32), 60, "eno4", "hll3", "fp64", "small tiles"),        # 600, fewer cells than 256^2
    (2, (256, 128), 1, "none", "central", "fp64", "small tiles"),    # 304
    (2, (240, 128), 1, "none", "central", "fp64", "faces"),          # 285
    (2, (256, 128), 1, "none", "central", "fp32", "faces"),
    (2, (640, 625), 1, "weno2", "hll3", "fp64", "small tiles"),      # 400,000 cells
    (2, (640, 626), 1, "weno2", "hll3", "fp64", "rows"),
    (2, (520, 520), 1, "weno2", "hll3", "fp32", "rows"),
    (2, (300, 300), 1, "none", "tecno1", "fp64", "tiles"),
    (2, (64, 64), 1, "none", "tecno4", "fp64", "tiles"),
    (3, (28, 28, 28), 1, "weno2", "hll3", "fp64", "faces"),          # 280
    (3, (33, 28, 28), 1, "weno2", "hll3", "fp64", "tiles"),          # 350
    (3, (24, 24, 24), 1, "eno3", "hll3", "fp64", "faces"),           # 144
    (3, (28, 28, 28), 1, "eno3", "hll3", "fp64", "tiles"),
    (3, (28, 28, 28), 1, "weno2", "hll3", "fp32", "tiles"),
    (3, (40, 40, 64), 1, "weno2", "hll3", "fp64", "tiles"),          # 400 tiles
    (3, (40, 41, 56), 1, "weno2", "hll3", "fp64", "columns"),        # 420, fewer cells
    (3, (50, 50, 41), 1, "eno3", "hll3", "fp64", "tiles"),
    (1, (1024,), 1, "weno2", "hll", "fp64", "lines"),
    (1, (1024,), 4096, "weno2", "hll", "fp64", "lines"),             # several rounds
    (1, (64,), 4096, "weno2", "hll", "fp64", "lines"),
    (1, (256,), 148, "weno2", "hll", "fp64", "lines"),               # one round
    (1, (256,), 4096, "weno2", "hll", "fp64", "tiles"),
    (1, (4096,), 1, "weno2", "hll", "fp64", "lines"),
    (1, (8192,), 1, "weno2", "hll", "fp64", "faces"),
    (1, (8192,), 1, "weno2", "hll", "fp32", "lines"),
    (1, (8193,), 1, "weno2", "hll", "fp32", "faces"),
    (1, (1024,), 1, "none", "tecno1", "fp64", "faces"),
]


@pytest.mark.parametrize("dim,n,members,recon,flux,precision,kernel", CHOICES,
                         ids=["%s-m%d-%s-%s-%s" % ("x".join(map(str, c[1])), c[2], c[3], c[4], c[5])
                              for c in CHOICES])
def test_chosen_kernel(dim, n, members, recon, flux, precision, kernel):
    with als.Simulator(dim, n, flux=flux, reconstruction=recon, precision=precision,
                       members=members) as sim:
        assert sim.kernels() == [kernel]


@pytest.mark.parametrize("integ,stages", [("rungekutta3", 3), ("rungekutta2", 2)])
def test_lines_are_accounted_and_timed_as_they_run(integ, stages):
    with als.Simulator(1, (500,), integrator=integ, cfl=0.4, end_time=10.0) as sim:
        sim.set_state(smooth_random_state(3, 1, (500,), 2))
        assert sim.kernels() == ["lines"] and sim.launches_per_step() == 1
        assert len(sim.profile_step()) == 1 and sim.info()["steps"] == 1
        before = sim.get_state()
        tuned = sim.tune(4)
        assert tuned["blocks_per_sm"] == 0 and tuned["ms_per_step"] > 0
        assert sim.info()["steps"] == 1
        np.testing.assert_array_equal(sim.get_state(), before)
    with als.Simulator(1, (9000,), integrator=integ, cfl=0.4, end_time=10.0) as sim:
        assert sim.launches_per_step() == stages and len(sim.profile_step()) == stages


def test_levels_on_different_kernels_take_a_launch_each():
    levels = [{"n": (64, 64), "members": 2}, {"n": (128, 128), "members": 1}]
    with als.Simulator(2, levels=levels) as sim:
        assert sim.kernels() == ["faces", "faces"] and sim.launches_per_step() == 3
        sim.set_tiles([0, 1])
        assert sim.kernels() == ["faces", "small tiles"] and sim.launches_per_step() == 6


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,members", [(1000, 1), (1000, 20), (1000, 60), (1000, 120), (1000, 400),
                                       (257, 400), (200, 900), (100, 3000), (3000, 70), (5000, 4), (5000, 60)])
def test_line_members_on_both_sides_of_the_rules(c_oracle, n, members, precision):
    """The last of many lines against the oracle (FP64) and against the same
    line alone, bit for bit, whatever the cluster or launch per stage."""
    st = smooth_random_state(5, 1, (n,), 2)
    states = np.broadcast_to(smooth_random_state(6, 1, (n,), 2), (members,) + st.shape).copy()
    states[-1] = st
    out = []
    for batch in (states, st[None]):
        with als.Simulator(1, (n,), cfl=0.4, end_time=1.0, max_steps=5, precision=precision,
                           members=len(batch)) as sim:
            sim.set_state(batch)
            sim.run()
            out.append(sim.get_state(len(batch) - 1, 1)[0])
    np.testing.assert_array_equal(out[0], out[1])
    if precision == "fp64":
        cfg = c_oracle.config(1, (n,), [0.0], [1.0], "hll3", "weno2", "rungekutta3", "periodic", 1.4)
        rc, expect, dts, steps, t = c_oracle.simulate(cfg, st, 0.4, 1.0, max_steps=5)
        np.testing.assert_array_equal(out[0], expect)
