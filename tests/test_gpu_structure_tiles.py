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
