"""Every answer of awe_batch_tune can be selected: the kernel of several steps a
launch comes back after a one-step one, with the same results."""
import ctypes as C

import numpy as np
import pytest

from helpers import ricker

pytestmark = pytest.mark.gpu
D, NT = 5.0, 50


def _batch(order):
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(order)
    shots = []
    for x0, nx in [(0, 70), (40, 90)]:
        sou = np.array([[(x0 + 0.5 * nx) * D, 45 * D]], np.float32)
        rec = np.stack([(x0 + np.linspace(1, nx - 2, 12)) * D, np.full(12, 50 * D)], 1).astype(np.float32)
        shots.append((x0, nx, sou, rec))
    desc = awe.make_desc(2, (100, 130), (D, D), (0.0, 0.0), NT, 0.005, nb=10, fdorder=order, dabc=1, expl=1,
                         precision=awe.FAST)
    b = awe.Batch(desc, shots)
    b.set_model((150 + 30 * rng.random((130, 100))).astype(np.float32))
    return b, [rng.standard_normal((NT, 12)).astype(np.float32) for _ in shots]


@pytest.mark.parametrize("order", [4, 8])
def test_tuned_kernel_is_selectable(order):
    import wavefield_imaging_gb300 as awe

    b, obs = _batch(order)
    wav = ricker(NT, 0.005)
    with b:
        kernel, grid = C.c_int(), C.c_int()
        assert awe.lib().awe_batch_tune(b._h, 3, C.byref(kernel), C.byref(grid)) == 0
        b.select(kernel.value)
        b.select(5)
        few = b.info
        assert few.launches_per_forward < NT
        d0, (g0, J0) = np.concatenate(b.forward(wav), 1), b.gradient(wav, obs)
        b.select(0)
        assert b.info.launches_per_forward == NT
        d1, (g1, J1) = np.concatenate(b.forward(wav), 1), b.gradient(wav, obs)
        b.select(5)
        assert (b.info.tile_z, b.info.tile_x, b.info.grid) == (few.tile_z, few.tile_x, few.grid)
        d2, (g2, J2) = np.concatenate(b.forward(wav), 1), b.gradient(wav, obs)
        for kernel in (-1, 6):
            with pytest.raises(awe.AweError) as e:
                b.select(kernel)
            assert e.value.status == 1
    assert np.abs(d0).max() > 0 and J0 == J1 == J2
    for a in (d1, d2):
        np.testing.assert_array_equal(a, d0)
    for a in (g1, g2):
        np.testing.assert_array_equal(a, g0)


def test_not_selectable_where_it_does_not_apply():
    import wavefield_imaging_gb300 as awe

    b, _ = _batch(10)
    with b, pytest.raises(awe.AweError) as e:
        b.select(5)
    assert e.value.status == 4
