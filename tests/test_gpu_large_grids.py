"""FP32 grids above the sizes where a launch changes its form: Newtonian runs of more than 300 000 cells, which take
three sweeps a step (smaller ones take fused steps), and black-hole grids of 2^19 cells and more."""
import numpy as np
import pytest

import cases
from conftest import bit_equal

pytestmark = pytest.mark.gpu

ABOVE = (547, 603)  # 329 841 cells: ragged rows, segments inside a row, columns past the last full pair


@pytest.fixture(scope="module")
def cg(cosmos_lib):
    import cosmos_gb300
    return cosmos_gb300


def newton(cg, shape, bc):
    return cg.Grid(cg.NEWTONIAN, shape, 1.0 / shape[1], 1.4, cg.FP32, bc)


@pytest.mark.parametrize("bc", [0, 1])
def test_tensor_map_staging_is_bit_identical(cg, bc):
    """Rows staged by one tensor-map copy (Y sweeps, the X sweep that reduces the CFL maximum) and by one copy per
    field give the same run."""
    s = cases.newton_state(np.random.default_rng(21), ABOVE)
    out = []
    try:
        for on in (True, False):
            cg.set_tensor_maps(on)
            g = newton(cg, ABOVE, bc)
            g.set_prim(s)
            g.run_begin(2, 0.8, 1e9, 0.0, 2, max_steps=9)
            g.run_steps(9)
            r = g.run_end()
            out.append((r.steps, r.t, g.get_prim()))
            g.close()
    finally:
        cg.set_tensor_maps(True)
    assert out[0][0] == out[1][0] == 9 and out[0][1] == out[1][1]
    assert bit_equal(out[0][2], out[1][2])


def test_chunk_replay_equals_single_steps(cg):
    """21 steps in one call (two graphs of eight and five of one) and in 21 calls; a run that ends inside a graph."""
    s = cases.newton_state(np.random.default_rng(12), ABOVE)
    out = []
    for calls in ([21], [1] * 21):
        g = newton(cg, ABOVE, 1)
        g.set_prim(s)
        g.run_begin(2, 0.8, 1e9, 0.0, 2, max_steps=21)
        for n in calls:
            g.run_steps(n)
        r = g.run_end()
        out.append((r.steps, r.t, g.get_prim()))
        g.close()
    assert out[0][0] == out[1][0] == 21 and out[0][1] == out[1][1]
    assert bit_equal(out[0][2], out[1][2])
    g = newton(cg, ABOVE, 1)
    g.set_prim(s)
    g.run_begin(2, 0.8, 1e9, 0.0, 2, max_steps=11)
    g.run_steps(16)
    assert g.run_end().steps == 11


def test_four_quadrant_error(cg, oracle):
    """The four-quadrant problem at 560^2, 30 steps, within the bounds stated for 128^2."""
    n = 560
    s = cases.four_quadrant(n, 2)
    g = newton(cg, (n, n), 1)
    g.set_prim(s)
    m0 = g.field_sums()
    r = g.solve(2, 0.9, 1e9, 0.0, 2, max_steps=30)
    got, m1 = g.get_prim(), g.field_sums()
    want, steps, _, _ = oracle.solve(0, s, 2, 1.0 / n, 0.9, 1e9, 0.0, 2, 1.4, 1, max_steps=30)
    assert r.steps == steps == 30
    assert np.abs(got[..., 0] - want[..., 0]).mean() < 1e-5 * np.abs(want[..., 0]).mean()
    assert abs(m1[0] - m0[0]) < 1e-6 * abs(m0[0]) and abs(m1[4] - m0[4]) < 1e-6 * abs(m0[4])


@pytest.mark.parametrize("lim", [0, 1, 2])
@pytest.mark.parametrize("shape", [(547, 548), (548, 548), (8, 37501), (3648, 57), (3649, 57), (10944, 8), (10945, 8)])
def test_run_equals_single_sweeps_on_both_sides(cg, shape, lim):
    """299 756 cells (fused steps), 300 304 and 300 008 (three sweeps); fused steps of four and six tiles per SM, and
    a row more: the run's steps are the single sweeps'."""
    s = cases.riemann(shape, 3 + lim)
    s[..., 0] += 0.4
    s[..., 4] += 0.3
    s[..., 1:4] *= 0.5
    s *= 1.0 + 0.01 * np.random.default_rng(9).standard_normal(s.shape)
    for bc in (0, 1):
        a, b = newton(cg, shape, bc), newton(cg, shape, bc)
        a.set_prim(s)
        r = a.solve(2, 0.9, 1e30, 0.2, lim, max_steps=4)
        b.set_prim(s)
        t = 0.0
        for it in range(4):
            dt = b.stable_dt(0.9, t, 1e30, it)
            b.sweep(0, 2, dt * 0.5, 0.2, lim)
            b.sweep(1, 2, dt, 0.2, lim)
            b.sweep(0, 2, dt * 0.5, 0.2, lim)
            t += dt
        assert r.steps == 4 and r.t == t and r.status == 0
        assert bit_equal(a.get_prim(), b.get_prim())
        a.close()
        b.close()


@pytest.mark.parametrize("above", [2.0, 0.0])
@pytest.mark.parametrize("shape", [(9, 58301), (58301, 9)])
def test_black_hole_operations(cg, shape, above):
    """524 709 cells, long along x and along y: source step and sweeps against the FP64 path, within the bounds stated
    for small grids; a hole whose horizon and excised cells lie at one end, states as there."""
    s = cases.gr_state(np.random.default_rng(3), shape)
    dx = 1.0 / 40
    hole = cg.BlackHoleSpacetime(0.1, 0.9, 0.09, 0.12, 0.0)

    def each(precision):
        g = cg.Grid(2, shape, dx, 5.0 / 3.0, precision, 0, hole, sr_c2p64_above=above)
        out = []
        for op in (lambda: g.rk_source(0.002, 0.0, 1), lambda: g.sweep(0, 2, 0.002, 0.0, 1),
                   lambda: g.sweep(1, 2, 0.002, 0.0, 1)):
            g.set_prim(s)
            op()
            out.append(g.get_prim())
        g.close()
        return out
    for k, (got, want) in enumerate(zip(each(cg.FP32), each(cg.FP64))):
        rel = (np.abs(got - want) / (np.abs(want) + 1e-3)).max(axis=-1)
        assert np.median(rel) < 1e-5 and (rel > 1e-3).mean() < 0.02, (k, np.median(rel), (rel > 1e-3).mean())
