"""FP64 sweeps on both sides of the sizes where their launch changes (cosmos_gb300/csrc/kernels_exact.cu): two
threads to a cell or interface on small grids, one on larger ones, and black-hole blocks of one and of
several lines, against the oracle: bit for bit (tolerance 0)."""
import numpy as np
import pytest

import cases
from test_gpu_amr import amr_state, check_invariants, run_amr
from test_gpu_exact_tiles import BH, bit_equal, sweeps

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cg(cosmos_lib):
    import cosmos_gb300
    return cosmos_gb300


# pairs: a block has 30 cells of a row, or 30 of each of four columns; then grids above five warps to an SM, X
# tiles of one warp (59 columns) and of four (130)
@pytest.mark.parametrize("system", [0, 1])
@pytest.mark.parametrize("shape", [(3,), (61,), (5, 2), (2, 29), (61, 31), (59, 61), (400, 59), (160, 130)])
def test_two_threads_to_a_cell(cg, oracle, system, shape):
    rng = np.random.default_rng(40 + system + shape[0])
    s = cases.state(system, rng, shape)
    if len(shape) == 2 and shape[0] > 100:  # values off the integer pipes' range too
        s[12, :, 1:4] *= 1e-90
        s[20, 30:40, 2] = 5e-324
        s[40, 7, 3] = -1e-200
    sweeps(cg, oracle, system, s, 0.0)


# one block, several lines to a block, lines cut in pieces, and (25 500 cells) one thread to an interface
@pytest.mark.parametrize("shape", [(2,), (17,), (500,), (2, 2), (2, 90), (90, 2), (40, 7), (150, 33), (17, 1500), (1500, 17)])
def test_black_hole_blocks(cg, oracle, shape):
    rng = np.random.default_rng(60 + shape[0])
    s = cases.state(2, rng, shape)
    sweeps(cg, oracle, 2, s, 0.0)
    hole = cg.BlackHoleSpacetime(*BH[2])
    g = cg.Grid(2, shape, 1.0 / 64, cases.SYS_GAMMA[2], cg.FP64, cg.BC_TRANSMISSIVE, hole)
    g.set_prim(s)
    g.rk_source(0.002, 0.0, 1)
    assert bit_equal(g.get_prim(), oracle.rk_source(s, 1.0 / 64, 0.002, 0.0, 1, cases.SYS_GAMMA[2], BH[2]))
    g.close()


@pytest.mark.parametrize("system", [0, 1])
def test_masked_levels_above_the_pair_sizes(cg, oracle, system):
    """The fine level of 320 x 310 cells is above twenty warps to an SM, the coarse one below."""
    shape, T = (160, 155), 0.004
    s = amr_state(shape, system, 12)
    n, nf, t, status, cp, fp, cf, ff = run_amr(cg, system, s, T, 3.0, 2)
    wn, wnf, wcp, wfp, wcf, wff = oracle.amr_level1(system, s, 1.0 / shape[-1], 0.9, T, 3.0, 2, cases.SYS_GAMMA[system])
    assert (n, nf) == (wn, wnf) and ff.any()
    assert bit_equal(cp.reshape(-1), wcp) and bit_equal(fp.reshape(-1), wfp)
    check_invariants(cf, ff)


@pytest.mark.parametrize("dims", [1, 2])
def test_refinement_threshold_to_the_last_bit(cg, oracle, dims):
    """Tolerances that equal a cell's gradient, one ulp to either side, and ones no gradient is compared with in the
    short form (zero, negative, tiny, huge)."""
    rng = np.random.default_rng(2)
    shape = (60,) if dims == 1 else (20, 31)
    s = cases.state(0, rng, shape)
    s.reshape(-1, 5)[7, 0] = 1e250
    dx = 1.0 / 37
    rho = s.reshape(-1, shape[-1], 5)[0, :, 0]
    tols = [0.0, -1.0, 1e-300, 1e300, np.inf]
    for j in (20, 21, 25):
        t = abs((rho[j] - rho[j - 1]) / dx)
        tols += [t, np.nextafter(t, 0.0), np.nextafter(t, np.inf)]
    g = cg.Grid(0, shape, dx, 1.4, cg.FP64, cg.BC_TRANSMISSIVE, None)
    g.set_prim(s)
    for tol in tols:
        c0 = np.ones(int(np.prod(shape)), np.uint8)
        f0 = np.zeros(c0.size * 2 ** dims, np.uint8)
        c, f = g.amr_flags(tol, c0, f0)
        wc, wf = oracle.amr_flags(0, s, dx, tol, 1.4, c0, f0, bh=None)
        assert np.array_equal(c, wc) and np.array_equal(f, wf), tol
    g.close()
