"""The fused time step on block shapes other than the usual two, with the
refined band against both walls: every class of
ghost cell (copies, both interpolations, walls, corners), whole and partial
warps, one and several gather rounds per thread. Bit for bit with the oracle
(tolerance 0, as every FP64 comparison of the two)."""
import pytest

import amrlbm
from amrlbm import AmrLbm
from oracle_lib import Oracle
from parity import compare_state

pytestmark = pytest.mark.gpu


def near_walls(nx, ny, levels, every):
    """A flat domain whose bubble nearly fills its height."""
    D = 2 ** levels
    width, height = 5 * nx * D, 3 * ny * D
    p = amrlbm.bubble_params(16, 16, levels, radius=0.42 * min(width, height), xc=0.5 * width,
                             yc=0.5 * height, rho_ratio=50.0, visc_ratio=50.0, eo=10.0, mo=1e-2,
                             gy=1e-7, regrid_every=every)
    p.nx, p.ny, p.nbx, p.nby = nx, ny, 5, 3
    p.max_blks = amrlbm.tree_blocks(5, 3, levels)
    return p


@pytest.mark.parametrize("nx,ny,levels,every", [
    (4, 4, 2, 2), (6, 4, 2, 3), (8, 8, 2, 1), (6, 10, 2, 2), (12, 10, 2, 3), (16, 16, 2, 2), (20, 8, 2, 2),
    (24, 16, 1, 2),
])
def test_block_shapes(nx, ny, levels, every):
    p = near_walls(nx, ny, levels, every)
    orc = Oracle(p)
    orc.initialize_rising_bubble()
    with AmrLbm(p) as gpu:
        gpu.initialize_rising_bubble()
        compare_state(gpu, orc)
        for steps in (5, 3):
            orc.main_loop(steps)
            gpu.main_loop(steps)
            gpu.sync()
            compare_state(gpu, orc)
