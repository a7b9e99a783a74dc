"""The TMA-staged 3D steps on levels with padded lines (n1 % 4 != 0) and at
orders 2 to 8: partial tiles and line ends off the 16-byte boundaries, grids
of one tile, sources next to the shell.  AWE_EXACT equals the oracle bit for
bit, AWE_FAST is within the parity tests' rel-L2 1e-5; the gradient of such
grids equals the one of the one-thread-per-cell kernels."""
import numpy as np
import pytest

from helpers import rel_l2, ricker, run_engine

pytestmark = pytest.mark.gpu
D = 5.0


def _case(n, nb, order, nt, fsrf=0, seed=5):
    rng = np.random.default_rng(seed + sum(n))
    vel = (168.0 + 20.0 * rng.random(n[::-1])).astype(np.float32)
    vel[:, :, : n[0] // 5] = 300.0
    f = [0.5, 0.4, 0.45]
    sou = np.array([[f[1] * (n[1] - 1) * D, f[2] * (n[2] - 1) * D, f[0] * (n[0] - 1) * D]], np.float32)
    rec = np.stack([rng.uniform(0, (n[k] - 1) * D, 11) for k in (1, 2, 0)], 1).astype(np.float32)
    par = dict(n=list(n), d=[D] * 3, o=[0.0] * 3, nb=nb, nt=nt, dt=0.005, fdorder=order, dabc=1, fsrf=fsrf, expl=1,
               jsnap=20)
    return par, vel, ricker(nt, 0.005), sou, rec


@pytest.mark.parametrize("order", [2, 4, 6, 8])
@pytest.mark.parametrize("n,nb,fsrf", [((16, 16, 16), 4, 0), ((61, 17, 19), 6, 1), ((54, 33, 13), 8, 0),
                                       ((115, 22, 27), 6, 0)])
def test_orders_and_line_lengths_vs_oracle(order, n, nb, fsrf):
    import wavefield_imaging_gb300 as awe
    from oracle import oracle
    from helpers import desc_from_par

    par, vel, wav, sou, rec = _case(n, nb, order, 60, fsrf)
    with awe.Plan(desc_from_par(par)) as p:
        assert p.step_kernel == "tma3d"
    ref, rsn = oracle.cart_cpu(par, vel, wav, sou, rec)
    assert np.abs(ref).max() > 0
    dat, snaps, _ = run_engine(par, vel, wav, sou, rec, precision=1)
    np.testing.assert_array_equal(dat, ref)
    np.testing.assert_array_equal(snaps.ravel(), rsn.ravel())
    # frames only: the longest grid's receivers see 1e-13 of the field in 60
    # steps, rounding residue that no FP32 kernel repeats to 1e-5
    _, snaps, _ = run_engine(par, vel, wav, sou, rec, precision=0)
    assert rel_l2(snaps.ravel(), rsn.ravel()) <= 1e-5


@pytest.mark.parametrize("order,n,fmt", [(2, (33, 21, 18), "BF16"), (4, (34, 20, 22), "BFP16"), (6, (35, 24, 20), "FP16"),
                                         (8, (37, 22, 20), "FP32")])
def test_gradient_of_padded_lines(monkeypatch, order, n, fmt):
    import wavefield_imaging_gb300 as awe
    from helpers import desc_from_par

    par, vel, wav, sou, rec = _case(n, 6, order, 50)
    out = []
    for kern in ("simple", ""):
        monkeypatch.setenv("AWE_STEP_KERNEL", kern)
        with awe.Plan(desc_from_par(par)) as p:
            p.set_model(vel)
            p.set_geometry(sou, rec)
            dobs = np.zeros((p.nsmp, len(rec)), np.float32)
            out.append(p.gradient(wav, dobs, ckpt_every=7, ckpt_format=getattr(awe, "CKPT_" + fmt)))
    assert np.abs(out[0][0]).max() > 0
    assert out[0][1] == out[1][1]
    np.testing.assert_array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("n,fsrf", [((95, 40, 33), 0), ((118, 30, 32), 1), ((57, 45, 46), 0)])
def test_shell_of_padded_lines(monkeypatch, n, fsrf):
    """Radius counts off a multiple of 4: traces, frames and gradient of the
    TMA kernels against the register marches."""
    import wavefield_imaging_gb300 as awe

    d, nt, nb = (0.005, 1.5e-6, 1.5e-6), 60, 8
    rng = np.random.default_rng(n[0])
    o = (3387.0, np.pi / 2 - (n[1] // 2) * d[1], -(n[2] // 2) * d[2])
    vel = (0.168 + 0.01 * rng.random(n[::-1])).astype(np.float32)
    sou = np.array([[o[0] + 0.6 * n[0] * d[0], o[2] + 0.4 * n[2] * d[2], o[1] + 0.5 * n[1] * d[1]]], np.float32)
    rec = np.array([[o[0] + 0.7 * n[0] * d[0], o[2] + k * d[2], o[1] + 0.45 * n[1] * d[1]]
                    for k in range(3, n[2] - 3, 4)], np.float32)
    wav, out = ricker(nt, 0.005), []
    for kern in ("simple", ""):
        monkeypatch.setenv("AWE_STEP_KERNEL", kern)
        desc = awe.make_desc(3, n, d, o, nt, 0.005, coords=awe.SPHER, scheme=awe.SCHEME_GPU, nb=nb, fsrf=fsrf, jsnap=20,
                             precision=awe.FAST)
        with awe.Plan(desc) as p:
            assert p.step_kernel == ("simple" if kern else "tma_sph")
            p.set_model(vel)
            p.set_geometry(sou, rec)
            dat, snaps = p.forward(wav, snapshots=True)
            g, J = p.gradient(wav, np.zeros_like(dat), ckpt_every=9, ckpt_format=awe.CKPT_FP32)
        out.append((dat, snaps, g))
    for a, b in zip(*out):
        assert np.abs(a).max() > 0 and rel_l2(b, a) <= 1e-6
