"""The FP64 primitive recovery and the black-hole state functions on conserved states as they come, physical or
not: the integer-pipe form against the hardware form against the reference's iteration (host build), and sweeps
over such cells against the oracle (GPU), bit for bit."""
import os
import subprocess

import numpy as np
import pytest

import cases

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_build_equals_reference(tmp_path):
    """300 k conserved states, among them tau = -D, S = 0, no root, negative D and tau, 60 decades off; as many
    black-hole states in and around the horizon."""
    exe = str(tmp_path / "exact_recovery_host")
    cpp = os.path.join(ROOT, "tests", "cpp")
    subprocess.run(["g++", "-O2", "-w", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(cpp, "host_cuda"), "-o", exe,
                    os.path.join(cpp, "exact_recovery_host.cpp")], check=True)
    r = subprocess.run([exe, "300000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def same(a, b):
    """The same bits, except that a NaN's sign and payload (which IEEE 754 leaves open) may be any."""
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(
        np.where(np.isnan(a), 0.0, a).view(np.uint64), np.where(np.isnan(b), 0.0, b).view(np.uint64))


def no_energy(shape, gamma):
    """Mild states, and cells at rest whose conserved energy tau + D is exactly zero: h = 1 + (p / rho) gamma /
    (gamma - 1) = -1 for rho = -1, p = 1, gamma = 2."""
    s = cases.sr_mild_state(np.random.default_rng(sum(shape)), shape)
    s.reshape(-1, 5)[7::29] = (-1.0, 0.0, 0.0, 0.0, 1.0)
    return s


# two threads to a cell; the wide X tiles; one dimension
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(33,), (20, 34), (160, 130)])
@pytest.mark.parametrize("gamma", [2.0, 1.0 + 2.0 ** -52, 1e20])
def test_sweeps_over_cells_without_energy(cosmos_lib, oracle, shape, gamma):
    """(2.0), and gammas beyond the integer pipes' bounds, where the hardware form takes every stage."""
    import cosmos_gb300 as cg
    s = no_energy(shape, gamma)
    for axis in range(len(shape)):
        for order in (1, 2):
            g = cg.Grid(1, shape, 1.0 / 64, gamma, cg.FP64, 0)
            g.set_prim(s)
            g.sweep(axis, order, 0.002, 0.0, 1)
            want = oracle.sweep(1, s, axis, order, 1.0 / 64, 0.002, 0.0, 1, gamma, 0)
            assert same(g.get_prim(), want), (axis, order)
            g.close()
