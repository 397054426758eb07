"""FP64 black-hole sweeps (cosmos_gb300/csrc/exact_tiles.cuh, gr_tile_kernel) over the block shapes that their rule
chooses: a line cut into pieces of 22 to 30 updates with a full or a short last one, two to seven short lines to a
block with lines left over, whole lines of 191, pieces of 287, both sides of the limit between two threads to an
interface and one; bit for bit with the oracle."""
import numpy as np
import pytest

import cases
from conftest import bit_equal

pytestmark = pytest.mark.gpu

# 24 320 cells (five warps to each of 152 SMs) end the form with two threads
SHAPES = [(190,), (191,), (192,), (382,), (383,), (24321,), (24710,), (3, 191), (2, 192), (192, 3), (193, 2), (9, 64),
          (64, 9), (127, 191), (128, 191), (193, 129), (65, 384), (384, 64)]


@pytest.mark.parametrize("shape", SHAPES)
def test_block_shapes(cosmos_lib, oracle, shape):
    import cosmos_gb300 as cg
    s = cases.gr_state(np.random.default_rng(sum(shape)), shape)
    dx = 1.0 / max(shape)
    for axis in range(len(shape)):
        for order in (1, 2):
            g = cg.Grid(2, shape, dx, 5.0 / 3.0, cg.FP64, 0, cg.BlackHoleSpacetime(*cases.GR_BH_SPIN))
            g.set_prim(s)
            g.sweep(axis, order, 0.1 * dx, 0.0, 1)
            want = oracle.sweep(2, s, axis, order, dx, 0.1 * dx, 0.0, 1, 5.0 / 3.0, bh=cases.GR_BH_SPIN)
            assert bit_equal(g.get_prim(), want), (axis, order)
            g.close()
