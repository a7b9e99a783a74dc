"""The cartesian and polar GPU-program steps in one launch at their edges: grids one block wide or
ending inside a block, sources at block edges and on the last line (where the
injection keeps its own launch), more sources than the step adds itself, a
graph replay and kept points.  AWE_EXACT equals the oracle bit for bit."""
import numpy as np
import pytest

from helpers import ricker

pytestmark = pytest.mark.gpu
D = 5.0


@pytest.mark.parametrize("kind,n,ns,edge", [
    ("cart2d", (12, 12), 1, False), ("cart2d", (48, 47), 3, False), ("cart2d", (49, 57), 8, False),
    ("cart2d", (60, 40), 9, False), ("cart2d", (50, 44), 2, True),
    ("polar2d", (48, 47), 3, False), ("polar2d", (49, 57), 9, False), ("polar2d", (40, 52), 2, True)])
def test_one_launch_step_is_bit_exact(kind, n, ns, edge):
    from oracle import oracle
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(n[0] + ns)
    polar, nb, nt = kind == "polar2d", 8, 50
    d = (0.005, 1e-4) if polar else (D, D)
    o = (3387.0, 1.5) if polar else (0.0, 0.0)
    unit = 1e-3 if polar else 1.0
    vel = ((150 + 30 * rng.random(n[::-1])) * unit).astype(np.float32)
    # axis positions in cells: block edges (64 and 8 padded cells) and, at the
    # edge, between the last two samples of the padded line
    c1 = rng.integers(1, max(n[0] - 2, 2), ns) + rng.choice([0.0, 0.25], ns)
    c2 = rng.integers(1, max(n[1] - 2, 2), ns) + rng.choice([0.0, 0.5], ns)
    if edge:
        (c1 if polar else c2)[0] = (n[0] if polar else n[1]) + nb - 1.5
    a1, a2 = o[0] + c1 * d[0], o[1] + c2 * d[1]
    sou = np.stack([a1, a2] if polar else [a2, a1], 1).astype(np.float32)
    r1, r2 = o[0] + rng.uniform(0, n[0] - 1, 9) * d[0], o[1] + rng.uniform(0, n[1] - 1, 9) * d[1]
    rec = np.stack([r1, r2] if polar else [r2, r1], 1).astype(np.float32)
    par = dict(kind=kind, n=list(n), d=list(d), o=list(o), nb=nb, nt=nt, dt=0.005, jsnap=20, bnds=1, fsrf=int(polar))
    wav = ricker(nt, 0.005)
    ref, rsn = oracle.gpu_scheme(kind, par, vel, wav, sou, rec)
    desc = awe.make_desc(2, n, d, o, nt, 0.005, coords=awe.SPHER if polar else awe.CART, scheme=awe.SCHEME_GPU,
                         nb=nb, jsnap=20, bnds=1, fsrf=polar, precision=awe.EXACT)
    with awe.Plan(desc) as p:
        p.set_model(vel)
        p.set_geometry(sou, rec)
        dat, snaps = p.forward(wav, snapshots=True)
        np.testing.assert_array_equal(dat, ref)
        np.testing.assert_array_equal(snaps, rsn)
        for _ in range(2):  # directly, captured, replayed; the same points set again
            np.testing.assert_array_equal(p.forward(wav), ref)
        p.set_geometry(sou, rec)
        np.testing.assert_array_equal(p.forward(wav), ref)


@pytest.mark.parametrize("n,n3,ns", [(12, 12, 2), (13, 15, 3), (33, 17, 8), (34, 44, 9), (45, 30, 2)])
def test_one_launch_step_3d_is_bit_exact(n, n3, ns):
    """Planes per block, face planes and shifted boundary lines; sources next
    to the boundary lines and on the padded faces."""
    from oracle import oracle
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(n + n3)
    nb, nt = 4, 40
    vel = (150 + 30 * rng.random((n3, n, n))).astype(np.float32)
    c = np.stack([rng.integers(0, q - 1, ns) + rng.choice([0.0, 0.5], ns) for q in (n, n3, n)], 1)
    c[0] = (-nb + 2.0, -nb + 5.5, -nb + 3.25)  # in the boundary shell
    sou = (c * D).astype(np.float32)
    rec = np.stack([rng.uniform(-nb, q + nb - 1.01, 12) * D for q in (n, n3, n)], 1).astype(np.float32)
    par = dict(kind="cart3d", n=[n, n, n3], d=[D] * 3, o=[0.0] * 3, nb=nb, nt=nt, dt=0.005, jsnap=15, bnds=1, jdata=2)
    wav = ricker(nt, 0.005)
    ref, rsn = oracle.gpu_scheme("cart3d", par, vel, wav, sou, rec)
    desc = awe.make_desc(3, (n, n, n3), (D,) * 3, (0.0,) * 3, nt, 0.005, scheme=awe.SCHEME_GPU, nb=nb, jsnap=15,
                         bnds=1, jdata=2, precision=awe.EXACT)
    with awe.Plan(desc) as p:
        p.set_model(vel)
        p.set_geometry(sou, rec)
        dat, snaps = p.forward(wav, snapshots=True)
        again = p.forward(wav)
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(dat, ref)
    np.testing.assert_array_equal(snaps, rsn)
    np.testing.assert_array_equal(again, ref)
