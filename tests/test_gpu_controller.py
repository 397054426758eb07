"""The device step controller (cosmos_gb300/csrc/device_common.cuh) as each kernel that enters a step compiles it."""
import math

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cg(cosmos_lib):
    import cosmos_gb300
    return cosmos_gb300


def grid(cg, kind, seed):
    """A run's grid: three FP64 sweeps a step, the fused FP32 step, three FP32 sweeps a step, one in 1D."""
    shape = {"fp64": (20, 33), "fused": (24, 57), "sweeps": (8, 37501), "line": (200,)}[kind]
    s = cases.newton_state(np.random.default_rng(seed), shape)
    dx = (0.7 + 0.01 * seed) / shape[-1]
    g = cg.Grid(cg.NEWTONIAN, shape, dx, 1.4, cg.FP64 if kind == "fp64" else cg.FP32, 1)
    return g, s, dx


def rule(g, s, dx, k):
    """Time before step k of a run from s, and its time step by the CFL rule (x0.2 up to step 6)."""
    g.set_prim(s)
    t = g.solve(2, 0.9, 1e30, 0.0, 1, max_steps=k - 1).t if k > 1 else 0.0
    dt = 0.9 * (dx / g.max_wavespeed())
    return t, dt * 0.2 if k <= 6 else dt


@pytest.mark.parametrize("kind", ["fp64", "fused", "sweeps", "line"])
def test_final_time_one_unit_below_a_step(cg, kind):
    """A final time one unit below the time that step k would reach shortens step k to the difference: the
    comparison of t + dt with the final time is of the rounded sum, in which dt is a rounded product."""
    for seed in range(6):
        g, s, dx = grid(cg, kind, seed)
        for k in range(1, 13):
            t, dt = rule(g, s, dx, k)
            end = math.nextafter(t + dt, 0.0)
            for final, last in ((1e30, t + dt), (t + dt, t + dt), (end, t + (end - t))):
                g.set_prim(s)
                r = g.solve(2, 0.9, final, 0.0, 1, max_steps=k)
                assert (r.steps, r.t) == (k, last), (seed, k, r.t, last)
        g.close()


def test_batch_final_time_one_unit_below_a_step(cg):
    """The same of the batch's controllers, against single grids of the same states."""
    for seed in range(6):
        grids = [grid(cg, kind, seed) for kind in ("fused", "line")]
        b = cg.Batch([s.shape[:-1] for _, s, _ in grids], [dx for _, _, dx in grids], 1.4, cg.FP32, 1)
        for k in range(1, 13):
            for m, (g, s, dx) in enumerate(grids):
                t, dt = rule(g, s, dx, k)
                end = math.nextafter(t + dt, 0.0)
                for final, last in ((1e30, t + dt), (t + dt, t + dt), (end, t + (end - t))):
                    for n, (_, q, _) in enumerate(grids):
                        b.set_prim(n, q)
                    b.run_begin(0.9, final, 0.0, 1, max_steps=k)
                    b.run_steps(k)
                    r = b.run_end()[m]
                    assert (r.steps, r.t) == (k, last), (seed, k, m, r.t, last)
        b.close()
