"""The one-launch ghost fill against the plain-C oracle's three passes (src/physics.hpp:354-432)
on random arrays, every value of every array: all boundary kinds per axis, 1-D to 3-D, extents
down to one above the ghost width (at it, a periodic pass reads a face that the same pass
writes). On the CPU the mapping itself (tests/bc_host.cu), on the GPU the
kernel."""
import ctypes as C
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle import portsim

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SHAPES = [(9, 1, 1, 3), (7, 5, 1, 3), (33, 4, 1, 2), (6, 5, 4, 3), (5, 4, 7, 3), (5, 6, 5, 4), (31, 3, 3, 2)]
FIELDS = ("u0", "b1f0", "b2f0", "b3f0")


def cases(shape):
    axes = [range(3) if n > 1 else (0,) for n in shape[:3]]
    return list(itertools.product(*axes))


def oracle_fill(shape, bc, rng):
    p = portsim.port_cfg()
    p.nx1, p.nx2, p.nx3, p.ng = shape
    for d in range(3):
        p.bc[d] = bc[d]
    p.x1max = p.x2max = p.x3max = 1.0
    p.recon, p.rsolver, p.nstage, p.gamma, p.cool_alpha = 2, 1, 3, 5.0 / 3.0, 1.0
    port = portsim.PortSim(p)
    before = {f: rng.normal(size=portsim.lib().port_size(port._h, f.encode())) for f in FIELDS}
    for f in FIELDS:
        port.set(f, before[f])
    portsim.lib().port_boundaries(port._h, 0)
    after = {f: port.get(f) for f in FIELDS}
    port.close()
    return before, after


@pytest.fixture(scope="module")
def host_fill(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("bc") / "bc_host.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(ROOT, "chasqui_b200", "csrc"), "-I", os.path.join(ROOT, "include"), "-o", so,
                    os.path.join(HERE, "bc_host.cu")], check=True, capture_output=True)
    return C.CDLL(so).fill


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_mapping_equals_the_three_passes(shape, host_fill):
    rng = np.random.default_rng(3)
    dp = C.POINTER(C.c_double)
    for bc in cases(shape):
        before, want = oracle_fill(shape, bc, rng)
        got = {f: np.ascontiguousarray(before[f]) for f in FIELDS}
        assert host_fill(*shape, (C.c_int * 3)(*bc), *[got[f].ctypes.data_as(dp) for f in FIELDS]) == 0
        for f in FIELDS:
            assert np.array_equal(got[f], want[f]), (bc, f, int((got[f] != want[f]).sum()))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_kernel_equals_the_three_passes(shape):
    from chasqui_b200 import Mesh, make_config
    rng = np.random.default_rng(4)
    for bc in cases(shape):
        before, want = oracle_fill(shape, bc, rng)
        m = Mesh(make_config(nx1=shape[0], nx2=shape[1], nx3=shape[2], nghost=shape[3], recon=2 if shape[3] > 2 else 1,
                             bc1=bc[0], bc2=bc[1], bc3=bc[2]))
        for f in FIELDS:
            m.set(f, before[f])
        m.boundaries(0)
        for f in FIELDS:
            assert np.array_equal(m.get(f).ravel(), want[f]), (bc, f)
        m.close()
