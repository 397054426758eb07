"""The FP64 operations on the integer pipes (cosmos_gb300/csrc/exact_math.cuh): their host build against
the machine's IEEE division, square root and product, bit for bit."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_build_equals_ieee(tmp_path):
    """3 M operand pairs over the fast range, its edges and the special values, each quotient and root
    with its FP32 estimate one unit low, exact and one unit high."""
    exe = str(tmp_path / "exact_math_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "exact_math_host.cpp")], check=True)
    r = subprocess.run([exe, "3000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_stages_equal_hardware_form(tmp_path):
    """300 k cell triples through the Newtonian and special-relativistic evolution and FORCE flux, all
    limiters, several biases, values up to and beyond the range: integer form = hardware form."""
    exe = str(tmp_path / "exact_stages_host")
    cpp = os.path.join(ROOT, "tests", "cpp")
    subprocess.run(["g++", "-O2", "-w", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(cpp, "host_cuda"), "-o", exe,
                    os.path.join(cpp, "exact_stages_host.cpp")], check=True)
    r = subprocess.run([exe, "300000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
