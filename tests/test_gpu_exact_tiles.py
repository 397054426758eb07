"""FP64 tile kernels (cosmos_gb300/csrc/exact_tiles.cuh) at the sizes where a tile, a warp or the choice
between the two tile widths ends, and on states that leave the integer pipes' range, against the
oracle: bit for bit (tolerance 0)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

BH = {0: None, 1: None, 2: cases.GR_BH_SPIN}
# X tiles update 30 or 126 cells (63 for the black hole), Y tiles 30 rows of 4 columns (31): one less, the
# tile, one more; 160 rows of 130 cells take the wide X tile, the others the narrow one
SHAPES = [(2,), (29,), (30,), (31,), (126,), (127,), (2, 63), (3, 64), (29, 5), (30, 4), (31, 3), (32, 2), (62, 9),
          (160, 130)]


@pytest.fixture(scope="module")
def cg(cosmos_lib):
    import cosmos_gb300
    return cosmos_gb300


def bit_equal(a, b):
    """The same bits, except that a NaN's sign and payload (which IEEE 754 leaves open) may be any."""
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(
        np.where(np.isnan(a), 0.0, a).view(np.uint64), np.where(np.isnan(b), 0.0, b).view(np.uint64))


def sweeps(cg, oracle, system, s, bias):
    gam, bh = cases.SYS_GAMMA[system], BH[system]
    hole = cg.BlackHoleSpacetime(*bh) if bh else None
    for axis in range(s.ndim - 1):
        for order, lim in ((1, 1), (2, 0), (2, 1), (2, 2)):
            for bc in ((0,) if system == 2 else (0, 1)):
                g = cg.Grid(system, s.shape[:-1], 1.0 / 64, gam, cg.FP64, bc, hole)
                g.set_prim(s)
                g.sweep(axis, order, 0.002, bias, lim)
                want = oracle.sweep(system, s, axis, order, 1.0 / 64, 0.002, bias, lim, gam, bc, bh=bh)
                assert bit_equal(g.get_prim(), want), (axis, order, lim, bc)
                g.close()


@pytest.mark.parametrize("system", [0, 1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_tile_edges(cg, oracle, system, shape):
    rng = np.random.default_rng(1000 * system + sum(shape))
    sweeps(cg, oracle, system, cases.state(system, rng, shape), 0.0)


@pytest.mark.parametrize("bias", [-1.0, -0.3, 0.4, 1.0])
def test_bias(cg, oracle, bias):
    """The limiter's general form (bias 0 has a shorter one)."""
    rng = np.random.default_rng(7)
    for system in (0, 1):
        sweeps(cg, oracle, system, cases.sr_mild_state(rng, (31, 33)), bias)


@pytest.mark.parametrize("system", [0, 1, 2])
def test_outside_the_integer_range(cg, oracle, system):
    """Cells whose values no integer-pipe operation takes (below 2^-255, above 2^257, subnormal, huge
    velocities' zeros) beside ordinary ones: the stages are formed again in hardware FP64."""
    rng = np.random.default_rng(11)
    s = cases.state(system, rng, (34, 67))
    s[5:9, 10:20, 1:4] = 0.0
    s[12, :, 1:4] *= 1e-90
    s[20, 30:40, 2] = 5e-324
    s[25, 7, 3] = -1e-200
    if system == 0:
        s[3, 40:50, [0, 4]] *= 1e-85
        s[28, 60:, [0, 4]] *= 1e90
    sweeps(cg, oracle, system, s, 0.0)
    g = cg.Grid(system, s.shape[:-1], 1.0 / 64, cases.SYS_GAMMA[system], cg.FP64, cg.BC_TRANSMISSIVE,
                cg.BlackHoleSpacetime(*BH[system]) if BH[system] else None)
    g.set_prim(s)
    assert g.max_wavespeed() == oracle.max_wavespeed(system, s, cases.SYS_GAMMA[system], bh=BH[system])
    if system == 2:
        g.rk_source(0.002, 0.0, 1)
        assert bit_equal(g.get_prim(), oracle.rk_source(s, 1.0 / 64, 0.002, 0.0, 1, cases.SYS_GAMMA[2], BH[2]))
