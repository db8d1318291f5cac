"""Batched cycles against the plain-C oracle, bit for bit but for the entropy (pow): members of
unequal extents and dimensions whose strong blasts are repaired (the bounded re-run of the update,
one march length for all members), and members with RKL2 diffusion whose stage counts differ."""
import numpy as np
import pytest

from chasqui_b200 import Batch, Mesh, make_config

SETS = {
    "fofc": [dict(n=(21, 17, 11)), dict(n=(45, 38, 1)), dict(n=(150, 1, 1)), dict(n=(40, 33, 37))],
    "one_large": [dict(n=(9, 8, 7)), dict(n=(72, 70, 66))],
    "rkl2": [dict(n=(17, 11, 9), nu=0.1, eta=0.2, sts=1), dict(n=(37, 22, 1), nu=0.4, eta=0.1, sts=1),
             dict(n=(13, 14, 15), eta=0.05, sts=1), dict(n=(20, 12, 1), kappa=0.3, sts=1)],
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SETS))
def test_batched_cycles_equal_the_oracle(name):
    from oracle import portsim
    rkl2 = name == "rkl2"
    cycles = 4 if name == "fofc" else 3
    meshes, ports = [], []
    for spec in SETS[name]:
        kw = {k: v for k, v in spec.items() if k != "n"}
        n = spec["n"]
        m = Mesh(make_config(nx1=n[0], nx2=n[1], nx3=n[2], x1min=-.5, x1max=.5, x2min=-.5, x2max=.5, x3min=-.5, x3max=.5,
                             cfl=0.4, tlim=10.0, **kw))
        if rkl2:
            m.init_problem("blast", [2.0, 0.5, 0.2, 0.5, 30.0, 1e-2, 11])
        else:
            m.init_problem("blast", [1e4, 1e-3, 0.2, 1.0, 30.0, 1e-2, 11])   # strong enough for repairs
        p = portsim.of_mesh(m)
        for f in ("u0", "b1f0", "b2f0", "b3f0"):
            p.set(f, m.get(f))
        m.prime(0.0)
        p.prime(0.0)
        p.cycles(cycles)
        meshes.append(m)
        ports.append(p)
    b = Batch(meshes)
    b.cycles(cycles)
    b.status()
    assert rkl2 or sum(m.counters()[0] for m in meshes) > 0
    bad = []
    for j, (m, p) in enumerate(zip(meshes, ports)):
        if m.clock()["t"] != p.clock()["t"] or (not rkl2 and m.counters()[0] != p.clock()["fofc"]):
            bad.append((j, "clock", m.clock()["t"], p.clock()["t"], m.counters()[0], p.clock()["fofc"]))
        for f in ("u0", "b1f0", "b2f0", "b3f0"):
            got, want = m.get(f).ravel(), p.get(f)
            if f == "u0":
                got, want = got.reshape(6, -1)[:5], want.reshape(6, -1)[:5]
            if not np.array_equal(got, want):
                bad.append((j, f, int((got != want).sum()), float(np.abs(got - want).max())))
    b.close()
    for m, p in zip(meshes, ports):
        p.close()
        m.close()
    assert not bad, bad
