"""Variable density in 3D: line lengths on and off the 16-byte boundaries, every
order up to 8.  AWE_EXACT equals the oracle bit for bit, AWE_FAST within rel-L2
1e-5; a model without a density after one with it runs at constant density
again."""
import numpy as np
import pytest

from helpers import desc_from_par, rel_l2, ricker, run_engine

pytestmark = pytest.mark.gpu


def _case(n1, order, nt=70):
    rng = np.random.default_rng(n1 + order)
    n, d = [n1, 26, 23], 5.0
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    den = (1.0 + 0.8 * rng.random(n[::-1])).astype(np.float32)
    sou = np.array([[0.4 * 25 * d, 0.5 * 22 * d, 0.5 * (n1 - 1) * d]], np.float32)
    rec = np.stack([rng.uniform(0, (n[a] - 1) * d, 15) for a in (1, 2, 0)], 1).astype(np.float32)
    par = dict(n=n, d=[d] * 3, o=[0.0] * 3, nb=8, nt=nt, dt=0.005, fdorder=order, dabc=1, expl=1, jsnap=30)
    return par, vel, den, ricker(nt, 0.005), sou, rec


@pytest.mark.parametrize("n1,order", [(28, 8), (29, 8), (28, 4), (30, 2), (28, 6)])
def test_density_vs_oracle(n1, order):
    from oracle import oracle

    par, vel, den, wav, sou, rec = _case(n1, order)
    ref, rsn = oracle.cart_cpu(par, vel, wav, sou, rec, den=den)
    plain, _ = oracle.cart_cpu(par, vel, wav, sou, rec)
    assert rel_l2(plain, ref) > 1e-2
    dat, snaps, _ = run_engine(par, vel, wav, sou, rec, den=den, precision=1)
    np.testing.assert_array_equal(dat, ref)
    np.testing.assert_array_equal(snaps.ravel(), rsn.ravel())
    _, snaps, _ = run_engine(par, vel, wav, sou, rec, den=den, precision=0)
    assert rel_l2(snaps.ravel(), rsn.ravel()) <= 1e-5


@pytest.mark.parametrize("n1", [28, 29])
def test_constant_density_after_a_variable_one(n1):
    import wavefield_imaging_gb300 as awe
    from oracle import oracle

    par, vel, den, wav, sou, rec = _case(n1, 8)
    plain, _ = oracle.cart_cpu(par, vel, wav, sou, rec)
    with awe.Plan(desc_from_par(par, precision=1)) as p:
        p.set_geometry(sou, rec)
        p.set_model(vel, den=den)
        assert p.step_kernel == "simple"
        for _ in range(3):  # launched, captured, replayed
            varied = p.forward(wav)
        p.set_model(vel)
        assert p.step_kernel == "tma3d"
        for _ in range(3):
            np.testing.assert_array_equal(p.forward(wav), plain)
    assert rel_l2(varied, plain) > 1e-2
