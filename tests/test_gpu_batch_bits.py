"""A member's result does not depend on the batch it runs in: the size rules
give a single small grid and a large batch of it different stage kernels, and
all of them give the same bits, in FP64 and in FP32 (whose contractions are
written out, csrc/euler_math.cuh).
"""
import numpy as np
import pytest

from oracle_lib import ghost_cells, smooth_random_state

torch = pytest.importorskip("torch")

import alsvinn_b200 as als  # noqa: E402

pytestmark = pytest.mark.gpu

RECONS = ["none", "weno2", "eno2", "eno3", "eno4", "mc", "mm", "wenof2", "weno3"]
SCHEMES = [(f, r) for f in ("hll3", "hll", "central") for r in RECONS] + \
    [("tecno1", "none"), ("tecno4", "none"), ("tecno6", "none")]
# a grid and the batch sizes that take it through the kernels of its dimension
GRIDS = [(1, (300,), (40, 200, 1500)), (2, (40, 36), (60, 130, 330)), (3, (12, 13, 11), (1, 14, 70))]


def _run(dim, n, flux, recon, integ, bc, precision, states, steps):
    with als.Simulator(dim, n, flux=flux, reconstruction=recon, integrator=integ, boundary=bc, cfl=0.3,
                       end_time=1e30, precision=precision, members=len(states)) as sim:
        sim.set_state(states)
        sim.advance(steps)
        last = len(states) - 1
        return sim.get_state(last, 1)[0], sim.info(last)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("dim,n,batches", GRIDS, ids=["1d", "2d", "3d"])
@pytest.mark.parametrize("flux,recon", SCHEMES, ids=["%s-%s" % s for s in SCHEMES])
def test_member_alone_and_in_batches(dim, n, batches, flux, recon, precision):
    g = ghost_cells(recon, flux)
    if any(v < 2 * g for v in n):
        pytest.skip("grid smaller than the stencil")
    for integ, bc in (("rungekutta3", "periodic"), ("rungekutta2", "neumann")):
        st = smooth_random_state(31 + len(recon), dim, n, g)
        alone, info = _run(dim, n, flux, recon, integ, bc, precision, st[None], 3)
        other = smooth_random_state(7, dim, n, g)
        for members in batches:
            states = np.broadcast_to(other, (members,) + other.shape).copy()
            states[-1] = st
            got, i = _run(dim, n, flux, recon, integ, bc, precision, states, 3)
            np.testing.assert_array_equal(got, alone)
            assert (i["t"], i["dt"]) == (info["t"], info["dt"])
