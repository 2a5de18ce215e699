"""The staged cube structure function (csrc/structure.cu) at its tiles' edges,
against the C oracle (agreement bar as in test_gpu_structure.py).
"""
import numpy as np
import pytest
import torch

from alsvinn_b200.functionals import structure_functions
from oracle_lib import smooth_random_state

pytestmark = pytest.mark.gpu


def _states(dim, n, g, members, seed):
    return np.stack([smooth_random_state(seed + m, dim, n, g) for m in range(members)])


@pytest.mark.parametrize("dim,n,members", [(2, (31, 75), 2), (2, (33, 4), 1), (2, (70, 130), 40),
                                           (3, (33, 9, 5), 2), (3, (12, 17, 10), 20)])
@pytest.mark.parametrize("bc", ["periodic", "neumann"])
@pytest.mark.parametrize("H", [1, 2, 6, 7, 8, 9])
def test_structure_cube_tile_edges(c_oracle, dim, n, members, bc, H):
    """Both sides of the largest H of the staged kernel (8 in 2-D, 6 in 3-D),
    tiles cut by the grid's end, tiles shared by several warps."""
    if dim == 3 and H > 7:
        H = 3
    st = _states(dim, n, 2, members, 31 * dim + H)
    out = structure_functions(torch.from_numpy(st).cuda(), dim, n, 2, bc, "cube", H, 1.0).cpu().numpy()
    for m in (0, members - 1):
        ref = c_oracle.structure_cube(dim, n, 2, bc, H, 1.0, st[m])
        np.testing.assert_allclose(out[m], ref, rtol=1e-12, atol=0)


@pytest.mark.parametrize("dim,n,members", [(2, (16, 16), 1), (2, (40, 37), 30), (2, (70, 64), 2), (3, (16, 9, 8), 1),
                                           (3, (20, 18, 17), 6)])
@pytest.mark.parametrize("bc", ["periodic", "neumann"])
@pytest.mark.parametrize("H,p", [(4, 2.5), (5, 0.5)])
def test_structure_cube_general_powers(c_oracle, dim, n, members, bc, H, p):
    """Powers that call pow, on both sides of the rule between the staged
    kernel and a thread per cell (pow is within 2 units in the last place of
    either library: 1e-12 as above)."""
    st = _states(dim, n, 2, members, 17 * dim + H)
    out = structure_functions(torch.from_numpy(st).cuda(), dim, n, 2, bc, "cube", H, p).cpu().numpy()
    for m in (0, members - 1):
        ref = c_oracle.structure_cube(dim, n, 2, bc, H, p, st[m])
        np.testing.assert_allclose(out[m], ref, rtol=1e-12, atol=0)
