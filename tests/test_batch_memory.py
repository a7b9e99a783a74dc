"""A batch gives back the memory of several steps a launch when something else
needs it: whatever fits with the one-step kernels fits, with the same traces and
gradient, before and after tuning; too little is an error every time."""
import numpy as np
import pytest

from helpers import ricker

pytestmark = pytest.mark.gpu
D, NT = 5.0, 40


def _survey():
    rng = np.random.default_rng(5)
    nz, nxm, shots, obs = 200, 420, [], []
    for x0, nx in [(0, 210), (100, 180), (180, 240)]:
        sou = np.array([[(x0 + 0.5 * nx) * D, 0.5 * nz * D]], np.float32)
        rec = np.stack([(x0 + np.linspace(1, nx - 2, 20)) * D, np.full(20, 0.5 * nz * D)], 1).astype(np.float32)
        shots.append((x0, nx, sou, rec))
        obs.append(rng.standard_normal((NT, 20)).astype(np.float32))
    return nz, nxm, (150 + 30 * rng.random((nxm, nz))).astype(np.float32), shots, obs


def _run(tune=False):
    """Traces and gradient, and what was raised; one retry of what failed."""
    import wavefield_imaging_gb300 as awe

    nz, nxm, vel, shots, obs = _survey()
    desc = awe.make_desc(2, (nz, nxm), (D, D), (0.0, 0.0), NT, 0.005, nb=10, fdorder=4, dabc=1, expl=1,
                         precision=awe.FAST)
    wav, out, bad = ricker(NT, 0.005), [], []
    try:
        with awe.Batch(desc, shots) as b:
            b.set_model(vel)
            for call in (lambda: np.concatenate(b.forward(wav), 1), lambda: b.gradient(wav, obs, ckpt_every=6)[0],
                         lambda: np.concatenate(b.forward(wav), 1), lambda: b.gradient(wav, obs, ckpt_every=6)[0]):
                try:
                    out.append(call())
                except awe.AweError as e:
                    bad.append(e.status)
            if tune:
                b.tune(3)
                out.append(np.concatenate(b.forward(wav), 1))
                out.append(b.gradient(wav, obs, ckpt_every=9)[0])
            launches = b.info.launches_per_forward
    except awe.AweError as e:
        return out, bad + [e.status], 0
    return out, bad, launches


def test_what_fits_one_step_a_launch_fits(monkeypatch):
    def fits(limit, kernel, tune=False):
        monkeypatch.setenv("AWE_STEP_KERNEL", kernel)
        monkeypatch.setenv("AWE_BATCH_BYTES_LIMIT", str(limit))
        return _run(tune)

    level = sum(nx + 20 for _, nx, _, _ in _survey()[3]) * 220 * 4
    want, bad, many = fits(0, "simple", True)
    assert not bad and many == NT
    free, bad, few = fits(0, "")
    assert not bad and few < NT
    lo, hi = 3 * level, 60 * level  # the least that the one-step kernels need
    while hi - lo > level // 16:
        mid = (lo + hi) // 2
        if fits(mid, "simple", True)[1]:
            lo = mid
        else:
            hi = mid
    for limit in [hi + k * level // 2 for k in range(0, 40, 3)]:
        out, bad, _ = fits(limit, "", True)
        assert not bad
        for a, b in zip(out[:4], want[:4]):
            np.testing.assert_array_equal(a, b)
        for a, b in zip(out[4:], want[4:]):
            assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()  # (the tuner's choice of kernel)
    for limit in (lo - 2 * level, lo - 8 * level):
        for kernel in ("simple", ""):
            out, bad, _ = fits(limit, kernel)
            assert bad and set(bad) == {3}  # AWE_ERR_NOMEM
            for a, b in zip(out[:1], want[:1]):
                np.testing.assert_array_equal(a, b)


def test_a_refused_selection_leaves_the_batch_usable(monkeypatch):
    """Items of another kernel that do not fit: an error, and the next runs use
    what the batch had, one step a launch if its extra memory was given back."""
    import wavefield_imaging_gb300 as awe

    nz, nxm, vel, shots, obs = _survey()
    desc = awe.make_desc(2, (nz, nxm), (D, D), (0.0, 0.0), NT, 0.005, nb=10, fdorder=8, dabc=1, expl=1,
                         precision=awe.FAST)
    wav = ricker(NT, 0.005)
    with awe.Batch(desc, shots) as b:
        b.set_model(vel)
        want, (grad, J) = np.concatenate(b.forward(wav), 1), b.gradient(wav, obs)
        assert np.abs(want).max() > 0
        for call in (lambda: b.select(4, chunk=1), lambda: b.select(3), lambda: b.tune(2)):
            monkeypatch.setenv("AWE_BATCH_BYTES_LIMIT", "1")
            with pytest.raises(awe.AweError) as e:
                call()
            assert e.value.status == 3
            np.testing.assert_array_equal(np.concatenate(b.forward(wav), 1), want)
            monkeypatch.delenv("AWE_BATCH_BYTES_LIMIT")
            g, J1 = b.gradient(wav, obs)
            np.testing.assert_array_equal(g, grad)
            assert J1 == J
