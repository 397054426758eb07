"""The FP32 special-relativistic primitive recovery against the reference's in FP64: the sweeps' iteration may
be no further off than the reference's own iteration in FP32, for a gas's states and for states that are none."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_build_no_further_off_than_the_reference_iteration(tmp_path):
    """20 k states of each of nine classes, gamma 1.1 to 3, the FP64 stage by Lorentz factor and always."""
    exe = str(tmp_path / "sr_recovery_host")
    cpp = os.path.join(ROOT, "tests", "cpp")
    subprocess.run(["g++", "-O2", "-w", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(cpp, "host_cuda"), "-o", exe,
                    os.path.join(cpp, "sr_recovery_host.cpp")], check=True)
    r = subprocess.run([exe, "20000"], capture_output=True, text=True)
    assert r.returncode == 0, "\n".join(line for line in r.stdout.splitlines() if line.endswith("<--"))
