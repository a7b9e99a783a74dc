"""awe_set_shots on small shells with an odd number of padded radii: every shot
is stepped, its traces those of a run of its own bit for bit, launched, captured
and replayed."""
import numpy as np
import pytest

from helpers import ricker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n3,nshots", [(39, 28, 3), (41, 20, 2), (37, 4, 4)])
def test_odd_radii_step_every_shot(n1, n3, nshots):
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(n1)
    n, d, nt = (n1, 30, n3), (0.005, 1.5e-6, 1.5e-6), 90
    o = (3387.0, np.pi / 2 - 15 * d[1], -(n3 // 2) * d[2])
    vel = (0.168 + 0.01 * rng.random(n[::-1])).astype(np.float32)
    wav = ricker(nt, 0.005)
    shots = []
    for k in range(nshots):
        sou = np.array([[o[0] + 25 * d[0], o[2] + (1 + k % n3) * d[2], o[1] + (14 + k) * d[1]]], np.float32)
        rec = np.array([[o[0] + 28 * d[0], o[2] + j * d[2] / 3, o[1] + (12 + k) * d[1]] for j in range(5 + k)], np.float32)
        shots.append((sou, rec))
    desc = awe.make_desc(3, n, d, o, nt, 0.005, coords=awe.SPHER, scheme=awe.SCHEME_GPU, nb=6, precision=awe.FAST)
    single = []
    with awe.Plan(desc) as p:
        assert p.npad[0] % 2 == 1
        p.set_model(vel)
        for s in shots:
            p.set_geometry(*s)
            single.append(p.forward(wav))
        p.set_shots(shots)
        for _ in range(3):
            together = p.forward(wav)
            off = 0
            for one in single:
                assert np.abs(one).max() > 0
                np.testing.assert_array_equal(together[:, off:off + one.shape[1]], one)
                off += one.shape[1]
