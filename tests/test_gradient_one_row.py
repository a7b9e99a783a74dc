"""The fold of the gradient onto models of one or two samples along axis 1, with
and without a free surface, whose zeroed samples are some of the only cell's
replicas: against the FP64 oracle."""
import numpy as np
import pytest

from helpers import desc_from_par, rel_l2, ricker

pytestmark = pytest.mark.gpu
D = 5.0


@pytest.mark.parametrize("n1", [1, 2, 3])
@pytest.mark.parametrize("fsrf", [0, 1])
def test_short_columns(n1, fsrf):
    import wavefield_imaging_gb300 as awe
    from oracle import oracle

    rng = np.random.default_rng(n1)
    n, nb, nt = (n1, 40), 8, 80
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    # (below the model: a free surface leaves nothing to inject into above)
    sou = np.array([[18.3 * D, (n1 + 1.4) * D]], np.float32)
    rec = np.stack([np.linspace(3, 36, 12) * D, np.full(12, (n1 + 2.2) * D)], 1).astype(np.float32)
    par = dict(n=list(n), d=[D, D], o=[0.0, 0.0], nb=nb, nt=nt, dt=0.005, fdorder=4, dabc=0, expl=1, fsrf=fsrf)
    wav, dobs = ricker(nt, 0.005), rng.standard_normal((nt, 12)).astype(np.float32)
    ref, _, _ = oracle.misfit_gradient(par, vel, wav, sou, rec, dobs)
    assert np.abs(ref).max() > 0
    with awe.Plan(desc_from_par(par)) as p:
        p.set_model(vel)
        p.set_geometry(sou, rec)
        g, _ = p.gradient(wav, dobs, ckpt_format=awe.CKPT_FP32)
    assert rel_l2(g, ref) <= 1e-4
