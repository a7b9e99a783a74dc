"""The gradient's source term at cells without a stencil (within nop of the
grid's edge), several steps a launch: sources in the padding of runs without a
sponge, outside the grid (all weight on the cell next to its first one) and on
the last sample of an axis.  Equal to the one-step kernels bit for bit."""
import numpy as np
import pytest

from helpers import desc_from_par, ricker

pytestmark = pytest.mark.gpu
D = 5.0


def _points(n, nb):
    """(x, z): on the outer cells of every side, outside the grid, on the last sample."""
    lo, mid = [-(nb - q) * D for q in (0.0, 0.4, 1.5)], [0.5 * (m - 1) * D for m in n]
    hi = [[(m + nb - 1 - q) * D for q in (0.2, 1.5)] for m in n]
    p = [(mid[1], q) for q in lo + hi[0]] + [(q, mid[0]) for q in lo + hi[1]] + [(lo[0], lo[1])]
    return p + [(-1e5, 0.0), (mid[1], (n[0] - 1) * D), ((n[1] - 1) * D, mid[0])]


@pytest.mark.parametrize("n,nb,order,dabc", [((70, 91), 4, 8, 0), ((121, 64), 5, 4, 0), ((64, 50), 3, 6, 0),
                                             ((90, 75), 1, 2, 0), ((80, 60), 4, 8, 1)])
def test_gradient_of_sources_at_the_edge(n, nb, order, dabc, monkeypatch):
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(nb)
    nt = 60
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    sou = np.array(_points(n, nb)[-2:] if dabc else _points(n, nb), np.float32)
    rec = np.stack([rng.uniform(-nb, n[1] + nb - 1.01, 60), rng.uniform(-nb, n[0] + nb - 1.01, 60)], 1) * D
    par = dict(n=list(n), d=[D, D], o=[0.0, 0.0], nb=nb, nt=nt, dt=0.005, fdorder=order, dabc=dabc, expl=1)
    dobs, out = rng.standard_normal((nt, 60)).astype(np.float32), []
    for kern in ("", "simple"):
        monkeypatch.setenv("AWE_STEP_KERNEL", kern)
        with awe.Plan(desc_from_par(par)) as p:
            p.set_model(vel)
            p.set_geometry(sou, rec.astype(np.float32))
            out.append([p.gradient(ricker(nt, 0.005), dobs, ckpt_every=e, ckpt_format=awe.CKPT_FP32)[0]
                        for e in (0, 13, 60)])
            few = p.last_launch_count()
        out[-1].append(few)
    assert out[0][-1] < out[1][-1]  # several steps a launch against one
    for a, b in zip(out[0][:-1], out[1][:-1]):
        assert np.isfinite(b).all() and np.abs(b).max() > 0
        np.testing.assert_array_equal(a, b)


def test_batch_gradient_of_sources_at_the_edge():
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(3)
    nz, nb, nt, windows, shots, obs = 72, 4, 50, [(0, 47), (20, 61)], [], []
    for x0, nx in windows:
        sou = np.array([(x + x0 * D, z) for x, z in _points((nz, nx), nb)], np.float32)
        rec = np.stack([(x0 + rng.uniform(0, nx - 1, 20)) * D, rng.uniform(0, nz - 1, 20) * D], 1).astype(np.float32)
        shots.append((x0, nx, sou, rec))
        obs.append(rng.standard_normal((nt, 20)).astype(np.float32))
    desc = awe.make_desc(2, (nz, 81), (D, D), (0.0, 0.0), nt, 0.005, nb=nb, fdorder=8, expl=1, precision=awe.FAST)
    with awe.Batch(desc, shots) as b:
        b.set_model((150 + 30 * rng.random((81, nz))).astype(np.float32))
        assert b.info.launches_per_forward < nt
        g0, _ = b.gradient(ricker(nt, 0.005), obs, ckpt_every=11, ckpt_format=awe.CKPT_FP32)
        b.select(0)
        g1, _ = b.gradient(ricker(nt, 0.005), obs, ckpt_every=11, ckpt_format=awe.CKPT_FP32)
    assert np.isfinite(g1).all() and np.abs(g1).max() > 0
    np.testing.assert_array_equal(g0, g1)
