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
