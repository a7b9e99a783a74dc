"""The TMA-marched 3D step at the plane counts where its chunk rule changes:
one item per column, a last chunk of one plane, chunks of eight planes, and
more than 64 planes.  AWE_EXACT equals the oracle bit for bit."""
import numpy as np
import pytest

from helpers import ricker, run_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3", [2, 8, 9, 49, 57, 58, 121])
def test_chunked_march_is_bit_exact(n3):
    from oracle import oracle

    rng = np.random.default_rng(n3)
    n, nb, nt = [24, 20, n3], 4, 30
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    sou = np.array([[47.0, 2.5 * (n3 - 1), 58.0]], np.float32)
    rec = np.stack([rng.uniform(5, 85, 20), rng.uniform(0, max(5.0 * (n3 - 1), 0.1), 20), rng.uniform(5, 105, 20)],
                   1).astype(np.float32)
    par = dict(n=n, d=[5.0] * 3, o=[0.0] * 3, nb=nb, nt=nt, dt=0.005, fdorder=8, dabc=1, expl=1)
    dat, _, _ = run_engine(par, vel, ricker(nt, 0.005), sou, rec, precision=1)
    ref, _ = oracle.cart_cpu(par, vel, ricker(nt, 0.005), sou, rec)
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(dat, ref)
