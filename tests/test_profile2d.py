"""Profiled 2D runs time the kernels that other runs launch: several steps a
launch, with the same launch counts and results."""
import numpy as np
import pytest

from helpers import desc_from_par, ricker

pytestmark = pytest.mark.gpu


def test_profiled_runs_take_several_steps_a_launch():
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(2)
    n, nt, d = (90, 110), 61, 5.0
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    sou = np.array([[54 * d, 40 * d]], np.float32)
    rec = np.stack([rng.uniform(0, 109, 30) * d, rng.uniform(0, 89, 30) * d], 1).astype(np.float32)
    par = dict(n=list(n), d=[d, d], o=[0.0, 0.0], nb=10, nt=nt, dt=0.005, fdorder=8, dabc=1, expl=1)
    wav, obs = ricker(nt, 0.005), rng.standard_normal((nt, 30)).astype(np.float32)
    with awe.Plan(desc_from_par(par)) as p:
        p.set_model(vel)
        p.set_geometry(sou, rec)
        dat, few = p.forward(wav), p.last_launch_count()
        g, _ = p.gradient(wav, obs, ckpt_every=9)
        few_g = p.last_launch_count()
        p.profile(True)
        dat1 = p.forward(wav)
        assert p.last_launch_count() == few < nt
        ms, launches = p.profile_read()
        assert launches == few and ms > 0
        g1, _ = p.gradient(wav, obs, ckpt_every=9)
        assert p.last_launch_count() == few_g
        kinds = p.profile_read_kinds()
        assert kinds["step"][1] >= 2 * few and few <= kinds["adjoint"][1] < nt
        assert kinds["step"][0] > 0 and kinds["adjoint"][0] > 0
    assert np.abs(g).max() > 0
    np.testing.assert_array_equal(dat1, dat)
    np.testing.assert_array_equal(g1, g)
