"""The device step controller's two forms in one run (host build)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_forms_of_a_step_in_any_order(tmp_path):
    """Ten steps, each by the time step kernel and sweeps or by a fused step: all 1024 orders."""
    exe = str(tmp_path / "controller_host")
    cpp = os.path.join(ROOT, "tests", "cpp")
    subprocess.run(["g++", "-O2", "-w", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(cpp, "host_cuda"), "-o", exe,
                    os.path.join(cpp, "controller_host.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
