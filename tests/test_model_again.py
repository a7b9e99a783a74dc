"""A new model on a plan refills its tables: the memory the plan holds stays the
same, and the run equals a new plan's."""
import numpy as np
import pytest

from helpers import ricker

pytestmark = pytest.mark.gpu


def test_models_on_one_cartesian_3d_gpu_program_plan():
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(4)
    n, d, nt = (24, 24, 20), 5.0, 40
    models = [(150 + 30 * rng.random(n[::-1])).astype(np.float32) for _ in range(3)]
    sou = np.array([[57.0, 48.0, 61.0]], np.float32)
    rec = rng.uniform(10, 90, (9, 3)).astype(np.float32)
    desc = awe.make_desc(3, n, (d,) * 3, (0.0,) * 3, nt, 0.005, scheme=awe.SCHEME_GPU, nb=8, precision=awe.FAST)
    wav, held = ricker(nt, 0.005), []
    with awe.Plan(desc) as p:
        p.set_geometry(sou, rec)
        for v in models:
            p.set_model(v)
            held.append(p.device_bytes())
            again = p.forward(wav)
    with awe.Plan(desc) as p:
        p.set_geometry(sou, rec)
        p.set_model(models[-1])
        new = p.forward(wav)
    assert np.abs(new).max() > 0
    np.testing.assert_array_equal(again, new)
    assert max(held[1:]) <= held[0] + 4 * nt + 4 * (nt + 1) * 9  # (the forward's staging buffers)
