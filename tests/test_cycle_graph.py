"""Cycles replayed from a captured graph, where the x sweep is a branch beside the y/z sweeps, end bit for
bit where launches one after the other end (per-kernel profiling keeps a mesh on those; a batch has
its own switch): FP64 and mixed, 1-D to 3-D, ragged, with repairs, on both sides of the branch's size rule."""
import numpy as np
import pytest

from chasqui_b200 import Batch, Mesh, make_config

pytestmark = pytest.mark.gpu
FIELDS = ("u0", "u1", "b1f0", "b2f0", "b3f0", "w", "f1", "f2", "e1", "e2", "e3")
SHAPES = [(130, 1, 1), (66, 35, 1), (257, 250, 1), (37, 9, 7), (61, 58, 63), (170, 165, 161)]


def mesh(n, precision, recon):
    m = Mesh(make_config(nx1=n[0], nx2=n[1], nx3=n[2], x1min=-.5, x1max=.5, x2min=-.5, x2max=.5, x3min=-.5, x3max=.5,
                         cfl=0.4, tlim=10.0, precision=precision, recon=recon))
    m.init_problem("blast", [1e4, 1e-3, 0.2, 1.0, 30.0, 1e-2, 11])   # strong enough for repairs
    m.prime(0.0)
    return m


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_replayed_cycles_equal_launches(shape, precision):
    recon = 2 if shape[0] != 61 else 3
    a, b = (mesh(shape, precision, recon) for _ in range(2))
    b.profile(True)
    for m in (a, b):
        m.cycles(5)
    assert a.clock() == b.clock() and a.counters() == b.counters()
    bad = [f for f in FIELDS if not np.array_equal(a.get(f), b.get(f), equal_nan=True)]
    a.close()
    b.close()
    assert not bad, bad


@pytest.mark.parametrize("precision", [0, 1])
def test_cycles_on_a_callers_stream_equal_replayed_ones(precision):
    """no graph there: the sweeps run side by side on the mesh's second stream, joined by events"""
    import ctypes
    import torch
    from chasqui_b200.core import load_library
    a, b = (mesh((66, 35, 1), precision, 2) for _ in range(2))
    c, d = (mesh((37, 40, 33), precision, 3) for _ in range(2))
    s = torch.cuda.Stream()
    for m in (b, d):
        for _ in range(3):
            assert load_library().chq_cycles(m._h, 2, ctypes.c_void_p(s.cuda_stream)) == 0
    s.synchronize()
    for x, y in ((a, b), (c, d)):
        x.cycles(6)
        assert x.clock() == y.clock()
        bad = [f for f in FIELDS if not np.array_equal(x.get(f), y.get(f), equal_nan=True)]
        x.close()
        y.close()
        assert not bad, bad


@pytest.mark.parametrize("precision", [0, 1])
def test_replayed_batches_equal_launches(precision):
    shapes = [(33, 30, 1), (20, 17, 11), (70, 1, 1), (41, 39, 40)]
    sets = [[mesh(s, precision, 2) for s in shapes] for _ in range(2)]
    for ms, graph in zip(sets, (True, False)):
        b = Batch(ms, graph=graph)
        b.cycles(5)
        b.status()
        b.close()
    bad = [(s, f) for s, x, y in zip(shapes, *sets) for f in FIELDS if not np.array_equal(x.get(f), y.get(f), equal_nan=True)]
    for m in sets[0] + sets[1]:
        m.close()
    assert not bad, bad
