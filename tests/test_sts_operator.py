"""RKL2 cycles against the plain-C oracle: state, clock and, after the last operator of a cycle,
the flux and edge-EMF arrays, for every set of diffusion coefficients (which decides the
components the operator touches), in 2-D and 3-D on ragged extents, with enough stages that the
state buffers rotate. FP64, bit for bit but for the entropy (pow), which nothing else reads."""
import numpy as np
import pytest

from chasqui_b200 import Mesh, make_config

COEF = {"nu": (0.2, 0.0, 0.0), "kappa": (0.0, 0.2, 0.0), "eta": (0.0, 0.0, 0.2), "nu_eta": (0.1, 0.0, 0.2),
        "all": (0.1, 0.2, 0.15)}
SHAPES = {"2d": (37, 22, 1), "3d": (17, 11, 9)}


@pytest.mark.gpu
@pytest.mark.parametrize("coef", sorted(COEF))
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_rkl2_cycles_equal_the_oracle(shape, coef):
    from oracle import portsim
    n1, n2, n3 = SHAPES[shape]
    nu, kappa, eta = COEF[coef]
    mesh = Mesh(make_config(nx1=n1, nx2=n2, nx3=n3, nu=nu, kappa=kappa, eta=eta, sts=1, tlim=10.0))
    port = portsim.of_mesh(mesh)
    mesh.init_problem("orszag_tang" if n3 == 1 else "cpaw", [2.0] if n3 == 1 else [1, 1, 1, 1.0, 0.3, 1.0, 0.2])
    for f in ("u0", "b1f0", "b2f0", "b3f0"):
        port.set(f, mesh.get(f))
    mesh.prime(0.0)
    port.prime(0.0)
    mesh.cycles(3)
    port.cycles(3)
    assert mesh.sts_stages() == port.sts_stages() and mesh.sts_stages() >= 9
    assert mesh.clock()["t"] == port.clock()["t"]
    bad = {}
    for f in ("u0", "b1f0", "b2f0", "b3f0", "f1", "f2", "f3", "e1", "e2", "e3"):
        got, want = mesh.get(f).ravel(), port.get(f)
        if f == "u0":
            got, want = got.reshape(6, -1)[:5], want.reshape(6, -1)[:5]
        if f == "f3" and n3 == 1:
            continue   # never written
        if not np.array_equal(got, want):
            bad[f] = (int((got != want).sum()), float(np.abs(got - want).max()))
    port.close()
    mesh.close()
    assert not bad, bad


@pytest.mark.gpu
def test_rkl2_scratch_is_four_states():
    """Y1, Y2, M0 and Mj, nine double components a frame point each: Y0 is u0 itself"""
    plain, sts = (Mesh(make_config(nx1=64, nx2=48, nx3=40, nu=0.1, sts=s)) for s in (0, 1))
    pitch = -(-(64 + 2 * plain.ng + 1) // 32) * 32
    points = -(-(40 + 2 * plain.ng + 1) * (48 + 2 * plain.ng + 1) * pitch // 64) * 64
    assert sts.nbytes - plain.nbytes == 36 * 8 * points
    for m in (plain, sts):
        m.close()
