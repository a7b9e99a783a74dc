"""Injection by cell (fixed sources, one thread per cell that sources touch):
coincident and overlapping sources with one series each must add up in the
(source, corner) order of the reference, bit for bit under AWE_EXACT."""
import numpy as np
import pytest

from helpers import ricker, run_engine

pytestmark = pytest.mark.gpu


def _points(rng, ns, n, nd):
    """ns source points around the middle, several of them on the same cells."""
    c = [0.5 * (k - 1) * 5.0 for k in (n[1], n[2] if nd == 3 else 1, n[0])]
    p = np.array([[q + 5.0 * rng.integers(-3, 4) + rng.choice([0.0, 1.25, 2.5]) for q in c] for _ in range(ns)])
    return (p if nd == 3 else p[:, [0, 2]]).astype(np.float32)


# 8 and 9: the last count added inside the 2D step kernel and the first beyond
# it; 130: more cells than one block of the list kernel
@pytest.mark.parametrize("nd,ns", [(2, 8), (2, 9), (2, 130), (3, 1), (3, 40)])
@pytest.mark.parametrize("each", [False, True])
def test_cpu_scheme_injection_is_bit_exact(nd, ns, each):
    from oracle import oracle

    rng = np.random.default_rng(ns + nd)
    n = [40, 44] if nd == 2 else [22, 24, 20]
    nt = 50
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    wav = ricker(nt, 0.005)
    if each:
        wav = (wav[:, None] * (0.5 + rng.random(ns))[None, :]).astype(np.float32)
    sou = _points(rng, ns, n, nd)
    rec = _points(rng, 12, n, nd)
    par = dict(n=n, d=[5.0] * nd, o=[0.0] * nd, nb=8, nt=nt, dt=0.005, fdorder=8, dabc=1, expl=0 if each else 1)
    dat, _, _ = run_engine(par, vel, wav, sou, rec, precision=1)
    ref, _ = oracle.cart_cpu(par, vel, wav, sou, rec)
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(dat, ref)


@pytest.mark.parametrize("ns,expl", [(1, 0), (33, 0), (33, 1)])
def test_gpu_scheme_injection_is_bit_exact(ns, expl):
    from oracle import oracle

    rng = np.random.default_rng(ns + expl)
    n, nt = [44, 52], 60
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    sou, rec = _points(rng, ns, n, 2), _points(rng, 9, n, 2)
    par = dict(kind="cart2d", n=n, d=[5.0, 5.0], o=[0.0, 0.0], nb=8, nt=nt, dt=0.005, jsnap=0, expl=expl)
    dat, _, _ = run_engine(par, vel, ricker(nt, 0.005), sou, rec, precision=1, scheme=0)
    ref, _ = oracle.gpu_scheme("cart2d", par, vel, ricker(nt, 0.005), sou, rec)
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(dat, ref)
