"""The branch-free quotients and roots of the flux kernel (chasqui_b200/csrc/chq_quot.cuh) give
the IEEE results over their stated ranges: built for the host with g++ (no contraction), the
hardware seeds emulated at their documented precision (tests/quot_check.cpp)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_quotients_equal_ieee(tmp_path):
    exe = tmp_path / "quot_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I",
                    os.path.join(ROOT, "chasqui_b200", "csrc"), "-o", str(exe), os.path.join(HERE, "quot_check.cpp")],
                   check=True)
    out = subprocess.run([str(exe), "2000000"], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
