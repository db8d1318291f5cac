"""Below 3-D a stage's corner EMFs and update run in one launch on small planes and in two on
large ones: whole cycles against the plain-C oracle on both sides of the size rule, 2-D and 1-D,
ragged, with FOFC repairs, state and edge EMFs bit for bit (the entropy's pow aside)."""
import numpy as np
import pytest

from chasqui_b200 import Mesh, make_config

#: extents and cycles; 2^18 points is the rule's line
SHAPES = {"33x47": (33, 47, 1, 4), "5x9": (5, 9, 1, 4), "97x5": (97, 5, 1, 4), "130": (130, 1, 1, 4),
          "513x511": (513, 511, 1, 1), "512x513": (512, 513, 1, 1)}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_cycles_below_3d_equal_the_oracle(name):
    from oracle import portsim
    n1, n2, n3, cycles = SHAPES[name]
    mesh = Mesh(make_config(nx1=n1, nx2=n2, nx3=n3, x1min=-.5, x1max=.5, x2min=-.5, x2max=.5, cfl=0.4, tlim=10.0))
    port = portsim.of_mesh(mesh)
    mesh.init_problem("blast", [1e4, 1e-3, 0.2, 1.0, 30.0, 1e-2, 11])   # strong enough for FOFC repairs
    for f in ("u0", "b1f0", "b2f0", "b3f0"):
        port.set(f, mesh.get(f))
    mesh.prime(0.0)
    port.prime(0.0)
    mesh.cycles(cycles)
    port.cycles(cycles)
    assert mesh.clock()["t"] == port.clock()["t"] and mesh.counters()[0] == port.clock()["fofc"]
    bad = {}
    for f in ("u0", "b1f0", "b2f0", "b3f0", "e1", "e2", "e3"):
        got, want = mesh.get(f).ravel(), port.get(f)
        if f == "u0":
            got, want = got.reshape(6, -1)[:5], want.reshape(6, -1)[:5]
        if not np.array_equal(got, want):
            bad[f] = (int((got != want).sum()), float(np.abs(got - want).max()))
    port.close()
    mesh.close()
    assert not bad, bad
