"""Fused FP32 steps (cosmos_gb300/csrc/step_tile.cuh): a run on a small grid against the same steps taken
sweep by sweep with the CFL rule's time step, bit for bit (the arithmetic per cell is the same)."""
import numpy as np
import pytest

import cases
from conftest import bit_equal

pytestmark = pytest.mark.gpu

# tiles are 56 columns x 12 rows with 4 and 2 of halo: one tile, its edges, a last column or row alone, odd widths
SHAPES = [(8, 8), (12, 56), (13, 57), (11, 55), (14, 58), (25, 113), (24, 112), (37, 170), (9, 59), (12, 61), (193, 257)]


@pytest.fixture(scope="module")
def cg(cosmos_lib):
    import cosmos_gb300
    return cosmos_gb300


@pytest.mark.parametrize("lim", [0, 1, 2])
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_equals_single_sweeps(cg, shape, bc, lim):
    s = cases.riemann(shape, 3 + lim)
    s[..., 0] += 0.4
    s[..., 4] += 0.3
    s[..., 1:4] *= 0.5
    s *= 1.0 + 0.01 * np.random.default_rng(9).standard_normal(s.shape)
    bias, dx, steps, t_final = 0.2, 1.0 / shape[1], 8, 1e30
    a = cg.Grid(cg.NEWTONIAN, shape, dx, 1.4, cg.FP32, bc)
    a.set_prim(s)
    r = a.solve(2, 0.9, t_final, bias, lim, max_steps=steps)
    b = cg.Grid(cg.NEWTONIAN, shape, dx, 1.4, cg.FP32, bc)
    b.set_prim(s)
    t = 0.0
    for it in range(steps):
        dt = b.stable_dt(0.9, t, t_final, it)
        b.sweep(0, 2, dt * 0.5, bias, lim)
        b.sweep(1, 2, dt, bias, lim)
        b.sweep(0, 2, dt * 0.5, bias, lim)
        t += dt
    assert r.steps == steps and r.t == t and r.status == 0
    assert bit_equal(a.get_prim(), b.get_prim())
    assert a.max_wavespeed() == b.max_wavespeed()


def test_end_of_run(cg):
    """Steps past the final time leave the grid as it is, a poisoned cell ends the run."""
    s = cases.smooth_state((40, 70), 1)
    g = cg.Grid(cg.NEWTONIAN, (40, 70), 1.0 / 70, 1.4, cg.FP32)
    g.set_prim(s)
    r = g.solve(2, 0.9, 0.02, 0.0, 1)
    end = g.get_prim()
    assert r.t == 0.02 and r.steps > 1
    g.set_prim(s)
    g.run_begin(2, 0.9, 0.02, 0.0, 1)
    g.run_steps(r.steps + 13)
    q = g.run_end()
    assert q.steps == r.steps and q.t == r.t and bit_equal(g.get_prim(), end)
    s[20, 30, 0] = np.nan
    g.set_prim(s)
    with pytest.raises(cg.CosmosError):
        g.solve(2, 0.9, 0.02, 0.0, 1)
