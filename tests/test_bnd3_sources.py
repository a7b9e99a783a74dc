"""Sources next to the cells that the 3D boundary launch rewrites: padding
between nop and 7 cells, sources zero to three cells from the first and last
model sample of every axis (among them on the last sample exactly, whose upper
corner has weight 0) and one outside the grid.  AWE_EXACT equals the oracle bit
for bit."""
import numpy as np
import pytest

from helpers import ricker, run_engine

pytestmark = pytest.mark.gpu
D = 5.0


def _run(n, nb, order, sou, nt=40):
    from oracle import oracle

    rng = np.random.default_rng(order + nb)
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    rec = np.stack([rng.uniform(0, (n[a] - 1) * D, 17) for a in (1, 2, 0)], 1).astype(np.float32)
    par = dict(n=list(n), d=[D] * 3, o=[0.0] * 3, nb=nb, nt=nt, dt=0.005, fdorder=order, dabc=1, expl=1, jsnap=13)
    wav = ricker(nt, 0.005)
    dat, snaps, _ = run_engine(par, vel, wav, sou, rec, precision=1)
    ref, rsn = oracle.cart_cpu(par, vel, wav, sou, rec)
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(dat, ref)
    np.testing.assert_array_equal(snaps.ravel(), rsn.ravel())


@pytest.mark.parametrize("n", [(30, 21, 19), (33, 22, 18)])  # at nb = 5, 7: padded lines whole and not
@pytest.mark.parametrize("order,nb", [(o, nb) for o in (2, 4, 6, 8) for nb in range(o // 2, 8)])
def test_sources_near_the_line_ends(n, order, nb):
    z = [q for k in (0.0, 1.0, 1.4, 2.3, 3.0) for q in (k, n[0] - 1 - k)]
    rng = np.random.default_rng(nb)
    sou = np.array([[rng.uniform(8, n[1] - 9) * D, rng.uniform(8, n[2] - 9) * D, q * D] for q in z], np.float32)
    _run(n, nb, order, sou)


@pytest.mark.parametrize("order,nb", [(4, 4), (8, 6), (8, 7)])
def test_corners_of_weight_zero_on_the_shell(order, nb):
    n = (34, 20, 22)
    mid = [0.5 * (n[a] - 1) * D for a in (1, 2, 0)]
    sou = []
    for k, a in enumerate((1, 2, 0)):  # (x, y, z) on the last sample of one axis
        p = list(mid)
        p[k] = (n[a] - 1) * D
        sou.append(p)
    sou.append([-100 * D, mid[1], mid[2]])  # outside the padded grid
    _run(n, nb, order, np.array(sou, np.float32))
