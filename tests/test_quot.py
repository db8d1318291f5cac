"""The branch-free quotients and roots of the flux kernel (chasqui_b200/csrc/chq_quot.cuh) give
the IEEE results over their stated ranges, divisors a few units from a power of two among them:
built for the host with g++ (no contraction), the hardware seeds emulated at their documented
precision (tests/quot_check.cpp), and on the device (tests/quot_device.cu)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_quotients_equal_ieee(tmp_path):
    exe = tmp_path / "quot_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-I",
                    os.path.join(ROOT, "chasqui_b200", "csrc"), "-o", str(exe), os.path.join(HERE, "quot_check.cpp")],
                   check=True)
    out = subprocess.run([str(exe), "2000000"], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr


@pytest.mark.gpu
def test_quotients_equal_ieee_on_the_device(tmp_path):
    exe = tmp_path / "quot_device"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-fmad=false", "-I",
                    os.path.join(ROOT, "chasqui_b200", "csrc"), "-o", str(exe), os.path.join(HERE, "quot_device.cu")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
