"""The face-flux kernels' branch-free solver against the plain-C oracle, bit for bit (FP64), on
states that reach each of its paths: ordinary shocks, gas at rest (both sides averaged), no
field (single-star region), supersonic flow, and states whose divisors leave the range of the
shared reciprocals, where the face is solved again with plain divisions, and a gas whose density,
sound speed and field are a few units from 1, where quotients lie closest to rounding midpoints. One
NaN cell must spread to the same faces, and so must velocities and fields that are infinite or whose
squares overflow, in isolated cells. Ragged extents leave partial warps, tiles and march segments."""
import numpy as np
import pytest

from chasqui_b200 import Mesh, make_config

SHAPES = {"3d": (37, 9, 7), "2d": (66, 35, 1), "1d": (130, 1, 1)}
SCHEMES = {"plm_hlld": (1, 1, 0), "ppm_hlld": (2, 1, 0), "wenoz_hlld": (3, 1, 0), "ppmx_lhlld": (4, 2, 0),
           "ppm_lhlld": (2, 2, 0), "plm_lhlld": (1, 2, 0), "ppm_hlld_char": (2, 1, 1), "wenoz_hlld_lowmach": (3, 1, 0)}
KINDS = ("random", "rest", "rest_noise", "no_field", "supersonic", "stiff", "out_of_range", "nan", "near_one", "overflow", "infinite")


def states(kind, shp, rng):
    """primitives (6), centred field (3) and face fields (3) on the padded arrays"""
    one = np.ones(shp)
    d, p = one.copy(), 0.1 * one
    v = [0.0 * one for _ in range(3)]
    b = [0.7 * one, 0.7 * one, 0.0 * one]
    if kind in ("random", "nan", "stiff", "out_of_range", "overflow", "infinite"):
        d, p = 1.0 + rng.random(shp), 0.1 + rng.random(shp)
        v = [rng.normal(size=shp) for _ in range(3)]
        b = [rng.normal(size=shp) for _ in range(3)]
    if kind == "rest_noise":
        d = 1.0 + 1e-3 * rng.random(shp)
    if kind == "no_field":
        d, v, b = 1.0 + rng.random(shp), [rng.normal(size=shp) for _ in range(3)], [0.0 * one] * 3
    if kind == "supersonic":
        v = [5.0 + rng.random(shp), -6.0 + rng.random(shp), 7.0 * one]
        d = 1.0 + 0.1 * rng.random(shp)
    if kind == "stiff":
        d, p = 10.0 ** rng.uniform(-8, 8, shp), 10.0 ** rng.uniform(-8, 8, shp)
    if kind == "out_of_range":
        far = rng.random(shp) < 0.2
        p = np.where(far, 1e120, p)
        d = np.where(rng.random(shp) < 0.1, 1e-9, d)
    if kind == "near_one":
        def near(a):
            return a + rng.integers(-4, 3, shp) * 2.0 ** -53
        d, p = near(1.0), near(0.6)
        v, b = [rng.integers(-2, 3, shp) * 2.0 ** -50 for _ in range(3)], [near(1.0), near(0.0), near(0.0)]
    b = [a.copy() for a in b]
    if kind in ("overflow", "infinite"):   # one component in every seventh cell of each axis
        k, j, i = np.indices(shp)
        lone = (i % 7 == 3) & ((j % 7 == 3) | (shp[1] == 1)) & ((k % 7 == 3) | (shp[0] == 1))
        big = rng.choice([1e80, 1e155, 1e160, -1e170] if kind == "overflow" else [np.inf, -np.inf], shp)
        pick = rng.integers(0, 5, shp)
        for q, a in enumerate(v + b[1:]):
            a[:] = np.where(lone & (pick == q), big, a)
    w = np.stack([d, v[0], v[1], v[2], p, p / d ** (5.0 / 3.0)])
    if kind == "nan":
        w[1, shp[0] // 2, shp[1] // 2, shp[2] // 2] = np.nan
    return w, np.stack(b)


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", sorted(SCHEMES))
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_fluxes_equal_the_oracle(shape, scheme):
    from oracle import portsim
    n1, n2, n3 = SHAPES[shape]
    recon, solver, char = SCHEMES[scheme]
    low = int(scheme.endswith("lowmach"))
    cfg = dict(nx1=n1, nx2=n2, nx3=n3, recon=recon, rsolver=solver, characteristic=char, low_mach=low)
    mesh = Mesh(make_config(**cfg))
    port = portsim.of_mesh(mesh)
    rng = np.random.default_rng(7)
    cells, faces = mesh.shape("w")[1:], mesh.shape("b1f0")[1:]
    dirs = [0] + [1] * mesh.two_d + [2] * mesh.three_d
    bad = []
    for kind in KINDS:
        w, b = states(kind, cells, rng)
        face = [np.zeros(faces) for _ in range(3)]
        for q in range(3):
            face[q][:cells[0], :cells[1], :cells[2]] = b[q]
        for name, a in [("w", w), ("bcc", b)] + [("b%df0" % (q + 1), face[q]) for q in range(3)]:
            mesh.set(name, a)
            port.set(name, a)
        mesh.fluxes_all(0)
        for d in dirs:
            portsim.lib().port_fluxes(port._h, d, 0)
        out = ["f%d" % (d + 1) for d in dirs] + ["e2x1", "e3x1"] + ["e1x2", "e3x2"] * mesh.two_d
        for f in out + ["e1x3", "e2x3"] * mesh.three_d:
            got, want = mesh.get(f).ravel(), port.get(f)
            if not np.array_equal(got, want, equal_nan=True):
                q = int(np.argmax((got != want) & ~(np.isnan(got) & np.isnan(want))))
                bad.append((kind, f, int((got != want).sum()), got[q], want[q]))
    port.close()
    mesh.close()
    assert not bad, bad


@pytest.mark.gpu
def test_cons_to_prim_next_to_one_equals_the_oracle():
    """densities (and, at rest, sound speeds) a few units from 1: velocities and the time step bit for bit"""
    from oracle import portsim
    mesh = Mesh(make_config(nx1=64, nx2=64, nx3=1, cfl=0.4))
    port = portsim.of_mesh(mesh)
    rng = np.random.default_rng(5)
    shp = mesh.shape("u0")
    u = np.zeros(shp)
    u[0] = 1.0 + rng.integers(-4, 3, shp[1:]) * 2.0 ** -53
    u[1:4] = rng.choice([0.0, 1.0, 0.5, 0.75], (3,) + shp[1:])
    u[4] = 0.9 + 0.5 * (u[1:4] ** 2).sum(0) / u[0]   # gamma p = 1
    for s in (mesh, port):
        s.set("u0", u)
        for q in (1, 2, 3):
            s.set("b%df0" % q, np.zeros(mesh.shape("b1f0")))
    dt, want = mesh.cons_to_prim(0, True), portsim.lib().port_cons_to_prim(port._h, 0, 1)
    got, exp = mesh.get("w"), port.get("w").reshape(mesh.shape("w"))
    port.close()
    mesh.close()
    assert dt == want
    assert np.array_equal(got[:5], exp[:5]), [int((got[n] != exp[n]).sum()) for n in range(5)]


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", ["plm_hlld", "ppm_hlld", "ppm_lhlld", "ppmx_lhlld"])
def test_mixed_fluxes_scale_with_the_units(scheme):
    """Single-precision fluxes of a gas in smaller units of mass (densities and pressures times 2^-s, fields
    times 2^-s/2, the same velocities) are the fluxes times 2^-s bit for bit: no face changes its
    arithmetic with the units. (Densities of 2^-40; at 2^-56 the product gamma p B^2 and its remainder of
    24 bits, 2^-112 B'^2 2^-24, are subnormal where the scaled field B' is small, in a few faces.)"""
    recon, solver, _ = SCHEMES[scheme]
    out = {}
    for s in (0, 20, 32, 40):
        mesh = Mesh(make_config(nx1=37, nx2=9, nx3=7, recon=recon, rsolver=solver, precision=1, dfloor=1e-30, pfloor=1e-30))
        rng = np.random.default_rng(11)
        cells, faces = mesh.shape("w")[1:], mesh.shape("b1f0")[1:]
        w, b = states("random", cells, rng)
        w[0], w[4], w[5], b = w[0] * 2.0 ** -s, w[4] * 2.0 ** -s, w[5], b * 2.0 ** (-s // 2)
        mesh.set("w", w)
        mesh.set("bcc", b)
        for q in range(3):
            face = np.zeros(faces)
            face[:cells[0], :cells[1], :cells[2]] = b[q]
            mesh.set("b%df0" % (q + 1), face)
        mesh.fluxes_all(0)
        out[s] = [mesh.get(f) * 2.0 ** s for f in ("f1", "f2", "f3")] + [mesh.get(f) * 2.0 ** (s // 2) for f in ("e2x1", "e3x1", "e1x2")]
        mesh.close()
    bad = [(s, q, int((a != b).sum())) for s in (20, 32, 40) for q, (a, b) in enumerate(zip(out[s], out[0])) if not np.array_equal(a, b)]
    assert not bad, bad
