"""Several 2D steps in one launch (overlapping tiles): grids of one tile, odd
sizes that end inside a strip of four cells, run lengths that are not a
multiple of the steps per launch, frames and decimated traces between, sources
on tile edges, more sources and receivers than threads of a block.  AWE_EXACT
equals the oracle, AWE_FAST the one-step kernel, bit for bit."""
import numpy as np
import pytest

from helpers import ricker, run_engine

pytestmark = pytest.mark.gpu


def _case(n, nb, order, nt, ns, nr, seed, **kw):
    rng = np.random.default_rng(seed)
    vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
    sou = np.stack([rng.uniform(0, n[1] - 1, ns), rng.uniform(0, n[0] - 1, ns)], 1) * 5.0
    rec = np.stack([rng.uniform(-nb, n[1] + nb - 1.01, nr), rng.uniform(-nb, n[0] + nb - 1.01, nr)], 1) * 5.0
    par = dict(n=list(n), d=[5.0, 5.0], o=[0.0, 0.0], nb=nb, nt=nt, dt=0.005, fdorder=order, dabc=1, expl=1, **kw)
    return par, vel, ricker(nt, 0.005), sou.astype(np.float32), rec.astype(np.float32)


CASES = [((9, 11), 4, 8, 40, 1, 5, {}), ((30, 41), 7, 8, 61, 3, 40, dict(fsrf=1)), ((50, 37), 10, 4, 62, 9, 700, {}),
         ((97, 130), 12, 4, 67, 300, 30, dict(jsnap=7)), ((101, 64), 9, 2, 63, 2, 30, dict(jsnap=25, bnds=1)),
         ((64, 250), 11, 6, 50, 2, 30, {}), ((300, 290), 10, 8, 45, 4, 60, {})]


@pytest.mark.parametrize("n,nb,order,nt,ns,nr,kw", CASES)
def test_exact_equals_the_oracle(n, nb, order, nt, ns, nr, kw):
    from oracle import oracle

    par, vel, wav, sou, rec = _case(n, nb, order, nt, ns, nr, n[0], **kw)
    dat, snaps, _ = run_engine(par, vel, wav, sou, rec, precision=1)
    ref, rsn = oracle.cart_cpu(par, vel, wav, sou, rec)
    assert np.abs(ref).max() > 0
    np.testing.assert_array_equal(dat, ref)
    if par.get("jsnap"):
        np.testing.assert_array_equal(np.asarray(snaps).ravel(), np.asarray(rsn).ravel())


@pytest.mark.parametrize("n,nb,order,nt,ns,nr,kw", CASES)
def test_fast_equals_the_one_step_kernel(n, nb, order, nt, ns, nr, kw, monkeypatch):
    par, vel, wav, sou, rec = _case(n, nb, order, nt, ns, nr, n[0], jdata=3, **kw)
    dat, snaps, few = run_engine(par, vel, wav, sou, rec)
    monkeypatch.setenv("AWE_STEP_KERNEL", "simple")
    ref, rsn, many = run_engine(par, vel, wav, sou, rec)
    assert few < many
    np.testing.assert_array_equal(dat, ref)
    if par.get("jsnap"):
        np.testing.assert_array_equal(snaps, rsn)


@pytest.mark.parametrize("n,nb,order,nt,ns,nr,kw", [
    ((30, 41), 7, 8, 61, 3, 40, dict(fsrf=1)), ((50, 37), 10, 4, 62, 9, 700, dict(jdata=2)),
    ((101, 64), 9, 2, 63, 2, 30, {}), ((150, 170), 10, 8, 45, 1, 60, {}), ((64, 250), 11, 6, 50, 2, 0, {})])
def test_gradient_and_image_equal_the_one_step_kernels(n, nb, order, nt, ns, nr, kw, monkeypatch):
    """The gradient's recompute and adjoint sweep several steps a launch, the
    imaging condition once per segment: the same bits as one step a launch,
    for one segment, segments of one step, and segments that end inside a launch."""
    import wavefield_imaging_gb300 as awe
    from helpers import desc_from_par

    par, vel, wav, sou, rec = _case(n, nb, order, nt, ns, nr, n[1], **kw)
    rng = np.random.default_rng(1)
    dobs = rng.standard_normal(((nt - 1) // par.get("jdata", 1) + 1, nr)).astype(np.float32)

    def run():
        out = []
        with awe.Plan(desc_from_par(par)) as p:
            p.set_model(vel)
            p.set_geometry(sou, rec)
            for every in (0, 1, 1000):
                g, J = p.gradient(wav, dobs, ckpt_every=every)
                out += [g, np.float64(J)]
            out.append(p.rtm(wav, dobs, awe.IMAGE_XCORR))
            out.append(p.rtm(wav, dobs, awe.IMAGE_BORN))
            p.profile(True)  # profiled runs go one step a launch: the lists of both forms
            out.append(p.gradient(wav, dobs)[0])
        return out

    ours = run()
    monkeypatch.setenv("AWE_STEP_KERNEL", "simple")
    for a, b in zip(ours, run()):
        np.testing.assert_array_equal(a, b)
    assert nr == 0 or np.abs(ours[0]).max() > 0


@pytest.mark.parametrize("nz,nb,order,windows,jdata,fsrf", [
    (12, 4, 2, [(0, 5), (3, 1)], 1, 0),            # windows narrower than a tile's strips
    (60, 10, 8, [(0, 47), (20, 90), (101, 33)], 3, 1),
    (120, 8, 4, [(0, 131), (7, 64), (7, 64)], 2, 0),  # two shots on one window
    (200, 20, 6, [(0, 129)], 1, 0)])
def test_batch_equals_the_tile_kernels(nz, nb, order, windows, jdata, fsrf):
    """Traces, misfit and gradient of several steps a launch over windows of
    several widths, against the one-step tile kernels (select(0)) bit for bit;
    segments and traces that end inside a launch."""
    import wavefield_imaging_gb300 as awe

    rng = np.random.default_rng(nz)
    nt, nxm = 53, max(x0 + nx for x0, nx in windows)
    vel = (150 + 30 * rng.random((nxm, nz))).astype(np.float32)
    shots = []
    for k, (x0, nx) in enumerate(windows):
        sou = np.stack([(x0 + rng.uniform(0.1, 0.9, k + 1) * (nx - 1)) * 5.0, rng.uniform(0.45, 0.6, k + 1) * (nz - 1) * 5.0], 1)
        rec = np.stack([(x0 + np.linspace(0, nx - 1, 9)) * 5.0, np.full(9, 0.5 * (nz - 1) * 5.0)], 1)
        shots.append((x0, nx, sou.astype(np.float32), rec.astype(np.float32)))
    desc = awe.make_desc(2, (nz, nxm), (5.0, 5.0), (0.0, 0.0), nt, 0.005, nb=nb, fdorder=order, dabc=1, expl=1,
                         jdata=jdata, fsrf=fsrf, precision=awe.FAST)
    wav, out = ricker(nt, 0.005), []
    # residuals at every receiver and step, whether the wave has come or not
    obs = [rng.standard_normal(((nt - 1) // jdata + 1, 9)).astype(np.float32) for _ in windows]
    with awe.Batch(desc, shots) as b:
        b.set_model(vel)
        assert b.info.launches_per_forward < nt
        for sel in (False, True):
            if sel:
                b.select(0)
                assert b.info.launches_per_forward == nt
            d = b.forward(wav)
            d2 = b.forward(wav)  # replayed
            g, J = b.gradient(wav, obs, ckpt_every=7, ckpt_format=awe.CKPT_FP32)
            out.append((d, d2, g, J))
    (d0, e0, g0, J0), (d1, e1, g1, J1) = out
    assert np.abs(g1).max() > 0 and J0 == J1
    for a, b_, c, e in zip(d0, d1, e0, e1):
        np.testing.assert_array_equal(a, b_)
        np.testing.assert_array_equal(c, e)
    # FP64 sums of the fold run in one order; the accumulators are the same bits
    np.testing.assert_array_equal(g0, g1)
