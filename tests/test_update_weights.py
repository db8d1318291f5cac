"""The update reads a register of zero weight through the other one: every pair of weights the
integrators use and each output register, registers that differ and hold infinities, against the
plain-C oracle (FP64, state and face fields bit for bit)."""
import numpy as np
import pytest

from chasqui_b200 import Mesh, make_config

WEIGHTS = [(1.0, 0.0, 1), (1.0, 0.0, 0), (0.0, 1.0, 1), (0.0, 1.0, 0), (0.75, 0.25, 1), (1.0 / 3.0, 2.0 / 3.0, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(17, 13, 11), (33, 47, 1), (130, 1, 1)])
def test_update_weights_equal_the_oracle(shape):
    from oracle import portsim
    mesh = Mesh(make_config(nx1=shape[0], nx2=shape[1], nx3=shape[2], cfl=0.3, tlim=10.0))
    port = portsim.of_mesh(mesh)
    mesh.init_problem("blast", [10.0, 0.1, 0.2, 1.0, 30.0, 1e-2, 11])
    for f in ("u0", "b1f0", "b2f0", "b3f0"):
        port.set(f, mesh.get(f))
    mesh.prime(0.0)
    port.prime(0.0)
    mesh.fluxes_all(0)
    mesh.corner_emf()
    for d in range(1 + mesh.two_d + mesh.three_d):
        portsim.lib().port_fluxes(port._h, d, 0)
    portsim.lib().port_corner_emf(port._h)
    rng = np.random.default_rng(3)
    regs = {f + "%d" % r: rng.normal(size=mesh.shape(f + "%d" % r)) for f in ("u", "b1f", "b2f", "b3f") for r in (0, 1)}
    for f in [f for f in regs if f[0] == "u"]:   # values that a product with zero would not leave alone
        regs[f][:, :, :, 6] = np.inf
        regs[f][:, :, :, 9] = -np.inf
    bad = {}
    for g0, g1, out in WEIGHTS:
        for f, a in regs.items():
            if g0 * g1 == 0.0 and f.endswith("1" if g1 == 0.0 else "0"):
                a = np.where(np.isfinite(a), a, 1.0)   # (the oracle multiplies the register of zero weight too)
            mesh.set(f, a)
            port.set(f, a)
        mesh.update(out, g0, g1, 1e-3)
        portsim.lib().port_update(port._h, out, g0, g1, 1e-3)
        for f in ("u%d", "b1f%d", "b2f%d", "b3f%d"):
            got, want = mesh.get(f % out).ravel(), port.get(f % out)
            if not np.array_equal(got, want, equal_nan=True):
                bad[(g0, g1, out, f)] = (int((got != want).sum()), float(np.abs(got - want).max()))
    port.close()
    mesh.close()
    assert not bad, bad
