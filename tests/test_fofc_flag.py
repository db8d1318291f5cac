"""The FOFC flag (with and without dual energy) and con2prim on states that have broken down, against the plain-C oracle: momenta
whose square, or whose kinetic energy, overflows, infinite and NaN components, densities and
pressures at and far below the floors, among ordinary cells."""
import numpy as np
import pytest

from chasqui_b200 import Mesh, make_config

INF, NAN = np.inf, np.nan
#: (density, m1, m2, m3, energy) of the broken cells
BROKEN = [(1.0, 1e160, 0.0, 0.0, 1.0), (1.0, 0.0, 2e154, 0.0, 1.0), (1e-9, 1e150, 1e150, 0.0, 1.0),
          (1e-5, 1e305 ** 0.5, 0.0, 0.0, 1.0), (1.0, INF, 0.0, 0.0, 1.0), (1.0, 0.0, -INF, 0.0, INF), (1.0, NAN, 0.0, 0.0, 1.0),
          (NAN, 1.0, 0.0, 0.0, 1.0), (INF, 1.0, 0.0, 0.0, 1.0), (1.0, 0.0, 0.0, 0.0, INF), (1.0, 0.0, 0.0, 0.0, -INF),
          (1.0, 0.0, 0.0, 0.0, NAN), (1e-10, 0.0, 0.0, 0.0, 1.0), (-1.0, 0.0, 0.0, 0.0, 1.0), (0.0, 1.0, 0.0, 0.0, 1.0),
          (1.0, 1.0, 1.0, 1.0, 1.5), (1e-300, 1e-200, 0.0, 0.0, 1e-30), (1e300, 1e150, 0.0, 0.0, 1.0), (1.0, 0.0, 0.0, 0.0, 1e308),
          (1e-9, 0.0, 0.0, 0.0, 1e307)]


@pytest.mark.gpu
@pytest.mark.parametrize("dual", [0, 1])
@pytest.mark.parametrize("shape", [(21, 9, 5), (65, 1, 1)], ids=str)
def test_broken_states_equal_the_oracle(shape, dual):
    from oracle import portsim
    mesh = Mesh(make_config(nx1=shape[0], nx2=shape[1], nx3=shape[2], dual_energy=dual))
    port = portsim.of_mesh(mesh)
    rng = np.random.default_rng(2)
    shp = mesh.shape("u1")
    u = np.empty(shp)
    u[0] = 1.0 + rng.random(shp[1:])
    u[1:4] = rng.normal(size=(3,) + shp[1:])
    u[4] = 4.0 + 0.5 * (u[1:4] ** 2).sum(0) / u[0]
    u[5] = 1.0
    cells = u.reshape(6, -1)
    active = np.flatnonzero(np.pad(np.ones(shape[::-1], bool), [(mesh.ng, mesh.ng) if n > 1 else (0, 0) for n in shape[::-1]]))
    at = rng.choice(active, len(BROKEN), replace=False)
    cells[:5, at] = np.array(BROKEN).T
    for s in (mesh, port):
        s.set("u1", u)
        for q in (1, 2, 3):
            s.set("b%df1" % q, np.zeros(mesh.shape("b1f1")))
    nbad, want = mesh.fofc_flag(1), portsim.lib().port_fofc_flag(port._h, 1)
    flag, wflag = mesh.get("flag").ravel()[active], port.get("flag")[active]
    wrong = [BROKEN[list(at).index(c)] if c in at else c for c in active[flag != wflag]]
    assert not wrong and nbad == want >= (4 if dual else 8), (wrong, nbad, want)
    if dual:
        port.close()
        mesh.close()
        return
    mesh.cons_to_prim(1, False)
    portsim.lib().port_cons_to_prim(port._h, 1, 0)
    bad = []
    for f in ("w", "u1"):
        a, b = mesh.get(f).reshape(6, -1)[:, active], port.get(f).reshape(6, -1)[:, active]
        same = np.array_equal(a[:4], b[:4], equal_nan=True)
        # the entropy goes through pow: the same infinities and NaNs, and close where finite
        near = np.isclose(a, b, rtol=1e-14, atol=0.0, equal_nan=True)
        if not (same and near.all()):
            c = int(np.argmin(near.all(axis=0)))
            bad.append((f, a[:, c], b[:, c]))
    port.close()
    mesh.close()
    assert not bad, bad
