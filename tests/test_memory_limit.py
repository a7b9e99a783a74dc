"""Memory that a plan can do without (the levels, slots and lists of several
steps a launch, the line-end copies and padded lines of a 3D level) is given back
when something else needs it: whatever fits with the one-step kernels fits, with
the same results.  Every limit in a process of its own (it is read once)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CODE = r'''
import sys; sys.path.insert(0, "."); sys.path.insert(0, "tests")
import hashlib
import numpy as np, wavefield_imaging_gb300 as awe
from helpers import ricker
kind = sys.argv[1]
n = dict(grad2d=(300, 290), frames2d=(300, 290), fwd3d=(70, 60, 52), shell=(101, 40, 40))[kind]
nt, d = 60, (5.0,) * len(n)
rng = np.random.default_rng(1)
vel = (150 + 30 * rng.random(n[::-1])).astype(np.float32)
axes = (1, 0) if len(n) == 2 else (1, 2, 0)
sou = np.array([[0.5 * (n[a] - 1) * 5.0 for a in axes]], np.float32)
rec = np.stack([rng.uniform(0, (n[a] - 1) * 5.0, 40) for a in axes], 1).astype(np.float32)
desc = awe.make_desc(len(n), n, d, (0.0,) * len(n), nt, 0.005, nb=10, fdorder=4, dabc=1, expl=1,
                     jsnap=10 if kind == "frames2d" else 0, precision=awe.EXACT if kind == "fwd3d" else awe.FAST)
res = []
def h(*a):
    return hashlib.sha1(b"".join(np.ascontiguousarray(x).tobytes() for x in a)).hexdigest()[:12]
def call(f):
    try:
        res.append(f())
    except awe.AweError as e:
        res.append("E%d" % e.status)
wav, obs = ricker(nt, 0.005), rng.standard_normal((nt, 40)).astype(np.float32)
if kind == "shell":  # r, theta, phi
    d = (0.005, 1.5e-6, 1.5e-6)
    o = (3387.0, np.pi / 2 - 20 * d[1], -20 * d[2])
    vel, axes = vel / 1000, (0, 2, 1)
    pt = lambda f: [o[a] + f * (n[a] - 1) * d[a] for a in axes]
    sou, rec = np.array([pt(0.5)], np.float32), np.array([pt(0.3 + 0.01 * k) for k in range(40)], np.float32)
    desc = awe.make_desc(3, n, d, o, nt, 0.005, coords=awe.SPHER, scheme=awe.SCHEME_GPU, nb=8, precision=awe.FAST)
held = launches = 0
try:
    p = awe.Plan(desc)
    p.set_model(vel); p.set_geometry(sou, rec)
    for _ in range(3):  # launched, captured, replayed
        if kind not in ("fwd3d", "shell"):
            call(lambda: h(p.gradient(wav, obs, ckpt_every=5)[0]))
            launches = p.last_launch_count()
        if kind == "frames2d":
            call(lambda: h(*p.forward(wav, snapshots=True)))
        if kind in ("fwd3d", "shell"):
            call(lambda: h(p.forward(wav)))
            launches = p.last_launch_count()
    held = p.device_bytes()
    if kind == "shell":
        res.append(p.step_kernel)
except awe.AweError as e:
    res.append("C%d" % e.status)
print(held, launches, " ".join(res))
'''


def _run(kind, limit=0, kernel=""):
    env = dict(os.environ, AWE_DEVICE_BYTES_LIMIT=str(limit) if limit else "", AWE_STEP_KERNEL=kernel)
    r = subprocess.run([sys.executable, "-c", _CODE, kind], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    held, launches, *res = r.stdout.strip().splitlines()[-1].split()
    return int(held), int(launches), res


@pytest.mark.parametrize("kind", ["grad2d", "frames2d", "fwd3d"])
def test_what_fits_one_step_a_launch_fits(kind):
    need, many, want = _run(kind, kernel="simple")
    level = {2: 320 * 310, 3: 90 * 80 * 72}[3 if kind == "fwd3d" else 2] * 4
    if kind == "frames2d":
        need += 6 * 300 * 290 * 4  # the frames' buffer of the call
    free, few, res = _run(kind)
    assert res == want and few < many and free > need - 2 * level
    top = max(free, need)
    for limit in (need, need + level // 2, need + 2 * level, need + 4 * level, (need + top) // 2, top + 8 * level):
        held, _, res = _run(kind, limit)
        assert res == want and held <= limit


def test_padded_lines_of_a_shell_give_way():
    need, _, want = _run("shell", kernel="simple")
    level = 117 * 56 * 56 * 4
    held, _, res = _run("shell", need)  # less than three padded levels
    assert need < 3 * level * 120 // 117 and held <= need
    assert res == want and res[-1] == "simple"
    _, _, res = _run("shell", need + level)
    assert res[-1] == "tma_sph" and not any(r.startswith(("E", "C")) for r in res)


def test_too_little_memory_is_an_error_every_time():
    need, _, want = _run("grad2d", kernel="simple")
    _, _, res = _run("grad2d", need - (1 << 19))
    assert set(res) == {"E3"} or res[0].startswith("C3")  # AWE_ERR_NOMEM
    assert len(want) == 3


_GEOMETRY = r'''
import sys; sys.path.insert(0, "."); sys.path.insert(0, "tests")
import numpy as np, wavefield_imaging_gb300 as awe
from helpers import ricker
shell = sys.argv[1] == "shell"
n = (40, 30, 28) if shell else (60, 50)
d = (0.005, 1.5e-6, 1.5e-6) if shell else (5.0, 5.0)
o = (3387.0, np.pi / 2 - 15 * d[1], -14 * d[2]) if shell else (0.0, 0.0)
desc = awe.make_desc(len(n), n, d, o, 40, 0.005, coords=awe.SPHER if shell else awe.CART,
                     scheme=awe.SCHEME_GPU if shell else awe.SCHEME_CPU, nb=6, dabc=not shell, expl=not shell)
axes = (0, 2, 1) if shell else (1, 0)
sou = np.array([[o[a] + 0.5 * n[a] * d[a] for a in axes]], np.float32)
rec = sou + np.array([2 * d[a] for a in axes], np.float32)
p, wav, res = awe.Plan(desc), ricker(40, 0.005), []
p.set_model(np.full(n[::-1], 0.168 if shell else 168.0, np.float32))
p.set_geometry(sou, rec)
ref = p.forward(wav)
many = np.repeat(sou, 400000, 0)
def call(f):
    try:
        f(); res.append(0)
    except awe.AweError as e:
        res.append(e.status)
for g in (lambda: p.set_geometry(many, rec), lambda: p.set_shots([(many, rec)] * 2) if shell else p.set_geometry(sou, many),
          lambda: p.set_moving_geometry(many, 400000, rec, 1)):
    call(g)
    call(lambda: p.forward(wav))
    call(lambda: p.gradient(wav, np.zeros((40, p.nr), np.float32)))
    p.set_geometry(sou, rec)
    assert np.array_equal(p.forward(wav), ref) and np.abs(ref).max() > 0
print(*res)
'''


@pytest.mark.parametrize("kind", ["plane", "shell"])
def test_points_that_do_not_fit_leave_no_half_set_geometry(kind):
    env = dict(os.environ, AWE_DEVICE_BYTES_LIMIT=str(8 << 20))
    r = subprocess.run([sys.executable, "-c", _GEOMETRY, kind], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    # AWE_ERR_NOMEM, then AWE_ERR_STATE until a geometry is set
    assert r.stdout.split() == ["3", "6", "6"] * 3
