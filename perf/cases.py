"""The measured work: forward modelling, gradients and surveys through the
package's public entry points (Plan, Batch), over the sizes and options that
programs use.

Every case is one dict of plain values:
  op       "forward" (Plan.forward_device), "gradient" (Plan.gradient_device),
           "survey" (Batch.forward_device), "survey_gradient" (Batch.gradient)
  program  "cpu": the 2N-order scheme of the cartesian CPU programs;
           "gpu": the scheme of the GPU programs (2nd order)
  coords   "cart", "polar" (2D) or "shell" (3D spherical)
  n1..n3   model samples (n3 = 0: 2D), nb padding, order, nt steps
  shots    shots of a survey or a shell track (1: one run)
  ns, nr   sources; receivers (per side of the receiver grid in 3D)
  each     one series per source (traces put back in at their receivers)
  free     free surface; den: variable density; precise: AWE_EXACT
  snap     steps between wavefield frames (0: none)
"""
import math

import numpy as np
import torch

import wavefield_imaging_gb300 as awe

DT = 0.005  # us
D = 5.0  # m (cartesian)


def _case(name, **kw):
    c = dict(op="forward", program="cpu", coords="cart", n1=0, n2=0, n3=0, nb=32, order=8, nt=100, shots=1, ns=1,
             nr=32, each=False, free=False, den=False, precise=False, snap=0)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a first look at a small section with the CPU program's default order: latency and launches
        _case("small_2d", n1=101, n2=143, nb=20, order=4, nt=300, nr=24),
        # the 512 x 512 sounding profile at 8th order, receivers at every column
        _case("profile_2d", n1=512, n2=512, nb=40, nt=1000, nr=512),
        # the GPU program's 2D run (2nd order, one-way boundary, free surface) on a section of odd size, a frame
        # every 100 steps
        _case("gpu_program_2d", program="gpu", n1=413, n2=587, nb=35, order=2, nt=500, nr=120, snap=100),
        # traces put back in at 601 receivers, one series each (the programs' adj=y)
        _case("back_injection_2d", n1=401, n2=603, nb=30, order=4, nt=300, ns=601, nr=64, each=True),
        # a stretch of a survey: 48 shots on windows of 300 to 700 columns, advanced together
        _case("survey_2d", op="survey", n1=512, n2=1200, nb=40, nt=150, shots=48, nr=128),
        # one FWI gradient of the profile, default checkpoints
        _case("gradient_2d", op="gradient", n1=512, n2=512, nb=40, nt=800, nr=512),
        # one FWI gradient of a stretch of the survey
        _case("survey_gradient_2d", op="survey_gradient", n1=512, n2=1000, nb=40, nt=100, shots=12, nr=128),
        # the 512^3 volume at 8th order, 128 x 128 receivers
        _case("volume_3d", n1=512, n2=512, n3=512, nb=32, nt=60, nr=128),
        # an ordinary volume of odd size with the CPU program's default order and a free surface,
        # with frames
        _case("volume_3d_o4", n1=201, n2=173, n3=149, nb=25, order=4, nt=150, nr=40, free=True,
              snap=50),
        # the GPU program's 3D cartesian run
        _case("gpu_program_3d", program="gpu", n1=150, n2=150, n3=133, nb=30, order=2, nt=120, nr=32),
        # four shots of a spherical-shell track advanced together, 64 x 64 receivers each
        _case("shell_track_3d", program="gpu", coords="shell", n1=350, n2=256, n3=256, nb=32, order=2, nt=50, shots=4,
              nr=64),
        # one FWI gradient of an ordinary volume, default checkpoints
        _case("gradient_3d", op="gradient", n1=160, n2=144, n3=150, nb=24, nt=60, nr=32),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["2d", "2d", "gpu2d", "back", "survey", "grad2d", "survey_grad", "3d", "3d", "gpu3d", "shell",
                       "grad3d"])
    if kind == "2d":
        return _case("", n1=_size(rng, 60, 1500), n2=_size(rng, 60, 2000), nb=rng.randint(10, 45),
                     order=rng.choice([2, 4, 6, 8, 8]), nt=_size(rng, 100, 1000), ns=rng.choice([1, 1, 3]),
                     nr=rng.randint(1, 500), free=rng.random() < 0.4, den=rng.random() < 0.15,
                     precise=rng.random() < 0.15, snap=rng.choice([0, 0, 0, 90]))
    if kind == "gpu2d":
        return _case("", program="gpu", coords=rng.choice(["cart", "cart", "polar"]), n1=_size(rng, 60, 1000),
                     n2=_size(rng, 60, 1200), nb=rng.randint(12, 45), order=2, nt=_size(rng, 100, 800),
                     ns=rng.choice([1, 1, 3]), nr=rng.randint(1, 400), free=rng.random() < 0.4,
                     precise=rng.random() < 0.15, snap=rng.choice([0, 0, 0, 90]))
    if kind == "back":
        dim3 = rng.random() < 0.4
        if dim3:
            return _case("", n1=_size(rng, 40, 160), n2=_size(rng, 40, 160), n3=_size(rng, 40, 160),
                         nb=rng.randint(10, 30), order=rng.choice([4, 8]), nt=_size(rng, 40, 150),
                         ns=rng.randint(20, 400), nr=rng.randint(4, 30), each=True)
        return _case("", n1=_size(rng, 100, 700), n2=_size(rng, 100, 700), nb=rng.randint(10, 40),
                     order=rng.choice([4, 8]), nt=_size(rng, 100, 500), ns=rng.randint(20, 700),
                     nr=rng.randint(1, 100), each=True)
    if kind in ("survey", "survey_grad"):
        op = "survey" if kind == "survey" else "survey_gradient"
        n1 = 4 * rng.randint(40, 160)
        shots = _size(rng, 2, 48 if op == "survey" else 14)
        return _case("", op=op, n1=n1, n2=_size(rng, 300, 1500), nb=2 * rng.randint(6, 20),
                     order=rng.choice([4, 8, 8]), nt=_size(rng, 50, 200 if op == "survey" else 110), shots=shots,
                     nr=rng.randint(16, 128), free=rng.random() < 0.3)
    if kind == "grad2d":
        return _case("", op="gradient", n1=_size(rng, 60, 700), n2=_size(rng, 60, 800), nb=rng.randint(10, 40),
                     order=rng.choice([4, 8, 8]), nt=_size(rng, 100, 700), nr=rng.randint(1, 400),
                     free=rng.random() < 0.3)
    if kind == "3d":
        return _case("", n1=_size(rng, 40, 280), n2=_size(rng, 40, 280), n3=_size(rng, 40, 280),
                     nb=rng.randint(8, 40), order=rng.choice([2, 4, 4, 6, 8, 8]), nt=_size(rng, 30, 120),
                     nr=rng.randint(2, 100), free=rng.random() < 0.4, den=rng.random() < 0.15,
                     precise=rng.random() < 0.15, snap=rng.choice([0, 0, 0, 25]))
    if kind == "gpu3d":
        n = _size(rng, 40, 220)  # the program asks for nx = nz
        return _case("", program="gpu", n1=n, n2=n, n3=_size(rng, 40, 220), nb=rng.randint(8, 35), order=2,
                     nt=_size(rng, 30, 120), nr=rng.randint(2, 60), precise=rng.random() < 0.15,
                     snap=rng.choice([0, 0, 0, 25]))
    if kind == "shell":
        op = rng.choice(["forward", "forward", "gradient"])
        return _case("", op=op, program="gpu", coords="shell", n1=2 * _size(rng, 30, 175), n2=_size(rng, 40, 220),
                     n3=_size(rng, 40, 220), nb=rng.randint(8, 32), order=2, nt=_size(rng, 30, 60),
                     shots=rng.choice([1, 1, 2, 4] if op == "forward" else [1, 1, 2]), nr=rng.randint(2, 64),
                     free=rng.random() < 0.4)
    return _case("", op="gradient", n1=4 * rng.randint(12, 40), n2=_size(rng, 48, 160), n3=_size(rng, 48, 160),
                 nb=2 * rng.randint(6, 14), order=rng.choice([4, 8, 8]), nt=_size(rng, 30, 70), nr=rng.randint(2, 40),
                 free=rng.random() < 0.3)


# ---- inputs (from the seed alone) ----

def _dims(c):
    return 3 if c["n3"] else 2


def _axes(c):
    """(n, d, o) of the model."""
    nd = _dims(c)
    n = (c["n1"], c["n2"], c["n3"])[:nd]
    if c["coords"] == "cart":
        return n, (D,) * nd, (0.0,) * nd
    d = (0.005, 0.04 / 512, 0.04 / 512)[:nd]  # km, rad
    o = (3387.0, math.pi / 2 - 0.5 * n[1] * d[1], -0.5 * c["n3"] * 0.04 / 512)[:nd]
    return n, d, o


def _model(c, seed):
    """Vacuum over ice with five dust layers over basalt with rough
    interfaces, [n3][n2][n1] (2D: [n2][n1]) float32, and a density if asked
    for.  m/us cartesian, km/us in the shell (vacuum at large radius)."""
    n, d, o = _axes(c)
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    n3 = n[2] if len(n) == 3 else 1
    unit = 1.0 if c["coords"] == "cart" else 1e-3
    depth = torch.arange(n[0], device="cuda", dtype=torch.float32) / n[0]
    if c["coords"] != "cart":
        depth = 1.0 - depth
    y = torch.arange(n3, device="cuda")[:, None] / 64.0
    x = torch.arange(n[1], device="cuda")[None, :] / 64.0
    rough = torch.zeros(n3, n[1], device="cuda")
    for _ in range(8):
        p = torch.rand(3, generator=g, device="cuda") * 6.28
        rough += torch.cos(p[0] * x + p[1] * y + p[2]) / 8
    surf = 0.15 + 0.03 * rough
    vel = torch.full((n3, n[1], n[0]), 168.0, device="cuda")
    for _ in range(5):
        r = torch.rand(3, generator=g, device="cuda").tolist()
        lo = (surf + 0.1 + 0.45 * r[0])[:, :, None]
        vel[(depth >= lo) & (depth < lo + 0.02 + 0.02 * r[1])] = 168.0 * (0.95 if r[2] < 0.5 else 1.05)
    vel[depth < surf[:, :, None]] = 300.0
    vel[depth >= (surf + 0.65)[:, :, None]] = 110.0
    vel *= (1 + 0.01 * torch.rand(vel.shape, generator=g, device="cuda")) * unit
    den = None
    if c["den"]:
        den = (1.0 + 0.5 * (vel < 250.0 * unit) + 0.1 * torch.rand(vel.shape, generator=g, device="cuda")).cpu().numpy()
    vel = vel.cpu().numpy()
    if _dims(c) == 2:
        return vel[0], None if den is None else den[0]
    return vel, den


def _points(c, seed, n2=None, x0=0):
    """Sources and receivers, (x, z), (x, y, z), (r, theta) or (r, phi, theta)."""
    rng = np.random.default_rng(int(seed) * 104729 + 5)
    n, d, o = _axes(c)
    n2 = n2 or n[1]
    z = [(0.1 if c["coords"] == "cart" else 0.9) * (n[0] - 1) + q for q in (0.3, 0.0)]
    az = [o[0] + q * d[0] for q in z]
    sx = x0 + (0.5 + (np.arange(c["ns"]) - 0.5 * (c["ns"] - 1)) * 0.9 / c["ns"]) * (n2 - 1) + 0.4 * rng.random(c["ns"])
    if len(n) == 2:
        rx = x0 + np.linspace(0.05, 0.95, c["nr"]) * (n2 - 1)
        if c["coords"] == "cart":
            s = np.stack([o[1] + sx * d[1], np.full(c["ns"], az[0])], 1)
            r = np.stack([o[1] + rx * d[1], np.full(c["nr"], az[1])], 1)
        else:
            s = np.stack([np.full(c["ns"], az[0]), o[1] + sx * d[1]], 1)
            r = np.stack([np.full(c["nr"], az[1]), o[1] + rx * d[1]], 1)
        return s.astype(np.float32), r.astype(np.float32)
    sy = 0.5 * (n[2] - 1) + rng.uniform(-0.2, 0.2, c["ns"]) * (n[2] - 1)
    gx, gy = np.meshgrid(np.linspace(0.3, 0.7, c["nr"]) * (n2 - 1), np.linspace(0.3, 0.7, c["nr"]) * (n[2] - 1),
                         indexing="ij")
    gx, gy = gx.ravel(), gy.ravel()
    if c["coords"] == "cart":
        s = np.stack([o[1] + sx * d[1], o[2] + sy * d[2], np.full(c["ns"], az[0])], 1)
        r = np.stack([o[1] + gx * d[1], o[2] + gy * d[2], np.full(gx.size, az[1])], 1)
    else:
        s = np.stack([np.full(c["ns"], az[0]), o[2] + sy * d[2], o[1] + sx * d[1]], 1)
        r = np.stack([np.full(gx.size, az[1]), o[2] + gy * d[2], o[1] + gx * d[1]], 1)
    return s.astype(np.float32), r.astype(np.float32)


def _ricker(nt, delay, f0=5.0):
    a = (math.pi * f0 * (np.arange(nt) * DT - delay)) ** 2
    return (1 - 2 * a) * np.exp(-a)


def _wavelet(c, seed):
    if not c["each"]:
        return _ricker(c["nt"], 0.15).astype(np.float32)[:, None]
    rng = np.random.default_rng(int(seed) * 31 + 1)
    t = np.arange(c["nt"])[:, None] * DT
    a = (math.pi * 5.0 * (t - (0.1 + 0.3 * rng.random(c["ns"]))[None, :])) ** 2
    return ((1 - 2 * a) * np.exp(-a) * (0.5 + rng.random(c["ns"]))[None, :]).astype(np.float32)


def _observed(c, seed, nrec):
    """Recorded traces [nt][nrec]: arrivals with a moveout."""
    rng = np.random.default_rng(int(seed) * 57 + 3)
    t = np.arange(c["nt"])[:, None] * DT
    off = np.abs(np.linspace(-1, 1, nrec))[None, :]
    out = np.zeros((c["nt"], nrec))
    for _ in range(3):
        t0, amp = rng.uniform(0.1, 0.8) * c["nt"] * DT, 0.05 * rng.uniform(0.3, 1.0)
        a = (math.pi * 5.0 * (t - np.sqrt(t0 ** 2 + (0.2 * c["nt"] * DT * off) ** 2))) ** 2
        out += amp * (1 - 2 * a) * np.exp(-a)
    return out.astype(np.float32)


def _windows(c, seed):
    """[(first column, columns)] of a survey's shots."""
    rng = np.random.default_rng(int(seed) * 13 + 7)
    hi = min(700, c["n2"])
    lo = max(60, min(300, hi // 2))
    out = []
    for _ in range(c["shots"]):
        nx = int(rng.integers(lo, hi + 1))
        out.append((int(rng.integers(0, c["n2"] - nx + 1)), nx))
    return out


def _inputs(c, seed):
    s = {"case": c, "wav": _wavelet(c, seed)}
    s["vel"], s["den"] = _model(c, seed)
    if c["op"].startswith("survey"):
        s["shots"] = [(x0, nx) + _points(c, seed + 1000 * k, nx, x0) for k, (x0, nx) in enumerate(_windows(c, seed))]
    else:
        s["shots"] = [(0, c["n2"]) + _points(c, seed + 1000 * k) for k in range(c["shots"])]
    if c["op"].endswith("gradient"):
        s["obs"] = [_observed(c, seed + k, q[3].shape[0]) for k, q in enumerate(s["shots"])]
    return s


def _desc(c):
    n, d, o = _axes(c)
    return awe.make_desc(len(n), n, d, o, c["nt"], DT, coords=awe.CART if c["coords"] == "cart" else awe.SPHER,
                         scheme=awe.SCHEME_CPU if c["program"] == "cpu" else awe.SCHEME_GPU, nb=c["nb"],
                         fdorder=c["order"], dabc=c["program"] == "cpu", fsrf=c["free"],
                         expl=c["program"] == "cpu" and not c["each"],
                         jsnap=c["snap"], precision=awe.EXACT if c["precise"] else awe.FAST)


def prepare(case, seed):
    s = _inputs(case, seed)
    c = case
    s["stream"] = torch.cuda.Stream()
    if c["op"].startswith("survey"):
        s["batch"] = b = awe.Batch(_desc(c), s["shots"])
        b.set_model(s["vel"])
        b.tune(5)
        if c["op"] == "survey":
            s["d_wav"] = torch.from_numpy(s["wav"]).cuda()
            s["d_dat"] = torch.zeros(b.info.total_samples, device="cuda")
    else:
        s["plan"] = p = awe.Plan(_desc(c))
        p.set_model(s["vel"], den=s["den"])
        if c["shots"] > 1:
            p.set_shots([q[2:] for q in s["shots"]])
        else:
            p.set_geometry(*s["shots"][0][2:])
        s["d_wav"] = torch.from_numpy(s["wav"]).cuda()
        if c["op"] == "gradient":
            s["d_obs"] = torch.from_numpy(np.ascontiguousarray(np.concatenate(s["obs"], 1))).cuda()
            s["d_grad"] = torch.zeros(s["vel"].shape, dtype=torch.float64, device="cuda")
        else:
            s["d_dat"] = torch.zeros(p.nsmp, p.nr, device="cuda")
            s["d_wfl"] = torch.zeros(p.nsnap, p.snap_elems, device="cuda")
    return s


def run(state):
    s, c = state, state["case"]
    if c["op"] == "survey_gradient":  # host buffers, as the entry point takes them
        return list(s["batch"].gradient(s["wav"], s["obs"]))
    st, here = s["stream"], torch.cuda.current_stream()
    st.wait_stream(here)
    wav, ncs = s["d_wav"].data_ptr(), s["wav"].shape[1]
    if c["op"] == "gradient":
        J = s["plan"].gradient_device(wav, ncs, s["d_obs"].data_ptr(), s["d_grad"].data_ptr(), stream=st.cuda_stream)
        out = [s["d_grad"], J]
    elif c["op"] == "survey":
        s["batch"].forward_device(wav, s["d_dat"].data_ptr(), stream=st.cuda_stream)
        out = [s["d_dat"]]
    else:
        wfl = s["d_wfl"].data_ptr() if c["snap"] else 0
        s["plan"].forward_device(wav, ncs, s["d_dat"].data_ptr(), wfl, stream=st.cuda_stream)
        out = [s["d_dat"], s["d_wfl"]] if c["snap"] else [s["d_dat"]]
    here.wait_stream(st)
    return out


def _cells(c):
    """Padded cells of all shots (survey windows: their mean width)."""
    p = [n + 2 * c["nb"] for n in _axes(c)[0]]
    if c["op"].startswith("survey"):
        hi = min(700, c["n2"])
        p[1] = (max(60, min(300, hi // 2)) + hi) // 2 + 2 * c["nb"]
    return c["shots"] * math.prod(p)


def work(case):
    """Per time step: both time levels and the squared velocity read and the
    new level written (16 bytes a cell); a gradient recomputes every step (20
    bytes with the stored level) and runs the adjoint step (36 bytes)."""
    c = case
    nd = _dims(c)
    flops = 3 * (c["order"] // 2) * nd * 2 + 6
    grad = c["op"].endswith("gradient")
    per = 72 if grad else 16
    steps = c["nt"] * _cells(c)
    model = 4 * math.prod(_axes(c)[0])
    traces = 4 * c["nt"] * c["shots"] * (c["nr"] ** 2 if nd == 3 else c["nr"])
    return {"bytes": steps * per + model + traces, "flops": steps * flops * (4 if grad else 1)}


# ---- the same in 64 bits, plain torch ----

F64 = dict(dtype=torch.float64, device="cuda")


def _interp(xs, oz, d, n):
    """Corner indices and weights along axes (z, x[, y]) in the order the
    coordinates are given; float32 as the coordinates come."""
    f32 = np.float32
    lo, fr = [], []
    inside = np.ones(xs[0].shape, bool)
    for x, o_, d_, n_ in zip(xs, oz, d, n):
        inside &= (x >= o_) & (x < f32(o_ + f32(f32(n_ - 1) * d_)))
    for k, (x, o_, d_) in enumerate(zip(xs, oz, d)):
        q = ((x - o_) / d_).astype(f32)
        j = np.where(inside, q.astype(np.int64), 0)
        lo.append(j)
        fr.append(np.where(inside, (q - j.astype(f32)).astype(np.float64), 1.0 if k == 0 else 0.0))
    return lo, fr


class _Grid:
    """Padded grid, tables and points of one shot in float64."""

    def __init__(self, c, vel, den, sou, rec, ox=0.0):
        f32 = np.float32
        n, d, o = _axes(c)
        nd, nb = len(n), c["nb"]
        self.c, self.nd, self.nb = c, nd, nb
        n = vel.shape[::-1]
        self.p = [q + 2 * nb for q in n]
        o = list(o)
        o[1] = f32(o[1]) + f32(ox)
        d32, o32 = [f32(q) for q in d], [f32(q) for q in o]
        opad = [f32(a - f32(f32(nb) * b)) for a, b in zip(o32, d32)]
        self.d, self.opad, self.dt = [float(q) for q in d32], opad, float(f32(DT))
        self.dt2 = float(f32(DT) * f32(DT))
        eps = f32(1e-4) if c["coords"] == "cart" and nd == 3 else f32(0)
        self.cut = [int(np.floor(f32(f32(a - q) / b) + eps)) if c["coords"] != "shell" else nb
                    for a, q, b in zip(o32, opad, d32)]
        self.idx = [torch.clamp(torch.arange(q, device="cuda") - nb, 0, m - 1) for q, m in zip(self.p, n)]
        self.v = self._pad(torch.from_numpy(vel).cuda().double())
        self.den = None if den is None else self._pad(torch.from_numpy(den).cuda().double())
        st = [1, self.p[0], self.p[0] * self.p[1]]

        def points(q):
            if c["coords"] == "cart":
                names = [0, 1] if nd == 2 else [0, 1, 2]  # z, x, y
                cols = [q[:, nd - 1], q[:, 0]] + ([q[:, 1]] if nd == 3 else [])
            else:  # z = theta (axis 2), x = r (axis 1), y = phi (axis 3)
                names = [1, 0] if nd == 2 else [1, 0, 2]
                cols = [q[:, nd - 1], q[:, 0]] + ([q[:, 1]] if nd == 3 else [])
            lo, fr = _interp(cols, [opad[a] for a in names], [d32[a] for a in names], [self.p[a] for a in names])
            ids, ws = [], []
            for k in range(1 << nd):
                i = sum((lo[a] + ((k >> a) & 1)) * st[names[a]] for a in range(nd))
                w = np.ones(len(q))
                for a in range(nd):
                    w = w * (fr[a] if (k >> a) & 1 else 1 - fr[a])
                ids.append(i)
                ws.append(w)
            return (torch.from_numpy(np.stack(ids, 1)).cuda(), torch.from_numpy(np.stack(ws, 1)).cuda())

        self.si, self.sw = points(sou)
        self.ri, self.rw = points(rec)
        (self._init_cpu if c["program"] == "cpu" else self._init_gpu)()

    def _pad(self, m):
        for a, i in enumerate(self.idx):
            m = m.index_select(m.ndim - 1 - a, i)
        return m.contiguous()

    def fold(self, g):
        """The transpose of the edge-replicating padding."""
        for a, i in enumerate(self.idx):
            dim = g.ndim - 1 - a
            shape = list(g.shape)
            shape[dim] = self.p[a] - 2 * self.nb
            g = torch.zeros(shape, **F64).index_add_(dim, i, g)
        return g

    def _sh(self, x, lo, k, axis):
        """Interior (lo cells from every face) of x shifted by k along axis."""
        s = []
        for a in reversed(range(self.nd)):
            q = k if a == axis else 0
            s.append(slice(lo + q, self.p[a] - lo + q))
        return x[tuple(s)]

    # the CPU programs' scheme
    def _init_cpu(self):
        c, h = self.c, self.c["order"] // 2
        f = math.factorial
        self.h = h
        self.cc = [0.0] + [-2.0 / (k * k) * math.cos(k * math.pi) * f(h) ** 2 / f(h + k) / f(h - k)
                           for k in range(1, h + 1)]
        self.W = torch.ones((), **F64)
        for a in range(self.nd):
            t = torch.ones(self.p[a], **F64)
            for i in range(min(self.nb, self.p[a])):
                t[i] = t[self.p[a] - 1 - i] = math.exp(-((self.nb - i - 1) / (math.sqrt(2.0) * 4 * self.nb)) ** 2)
            self.W = self.W * t.reshape([-1] + [1] * a)
        self.vel2 = self.v * self.v * self.dt2
        if c["free"]:
            self.vel2[..., : self.nb + 1] = 0
        self.abc = []
        if self.nd == 3:
            for a in range(3):
                for face in (self.nb, self.p[a] - self.nb - 1):
                    q = self.v.select(2 - a, face) * self.dt / self.d[a]
                    self.abc.append((1 - q) / (1 + q))

    def _lap(self, u):
        c0 = -2.0 * sum(self.cc) * sum(1.0 / d ** 2 for d in self.d)
        out = self._sh(u, self.h, 0, 0) * c0
        for a in range(self.nd):
            for k in range(1, self.h + 1):
                out = out + (self._sh(u, self.h, -k, a) + self._sh(u, self.h, k, a)) * (self.cc[k] / self.d[a] ** 2)
        if self.den is not None:
            dot = 0.0
            for a in range(self.nd):
                du = dr = 0.0
                for k in range(1, self.h + 1):
                    b = self.cc[k] * k / 2 / self.d[a]
                    du = du + (self._sh(u, self.h, k, a) - self._sh(u, self.h, -k, a)) * b
                    dr = dr + (self._sh(self.den, self.h, k, a) - self._sh(self.den, self.h, -k, a)) * b
                dot = dot + du * dr
            out = out - dot / self._sh(self.den, self.h, 0, 0)
        return out

    def _step_cpu(self, prv, cur, vel2, wav):
        """(levels before the step) -> (new level, the traces of cur)."""
        old = prv * self.W
        new = old.clone()
        inner = tuple(slice(self.h, q - self.h) for q in reversed(self.p))
        new[inner] = 2 * cur[inner] - old[inner] + vel2[inner] * self._lap(cur)
        new = self._inject(new, wav, vel2)
        if self.nd == 3:
            h = self.h
            for a in range(3):
                dim, m = 2 - a, self.p[a]
                for side in (0, 1):
                    if a == 0 and side == 0 and self.c["free"]:
                        continue
                    b = self.abc[2 * a + side]
                    for j in range(h):
                        i, q = (h - j, h - j + 1) if side == 0 else (m - h + j - 1, m - h + j - 2)
                        new.select(dim, i).copy_(cur.select(dim, q)
                                                 + (cur.select(dim, i) - new.select(dim, q).clone()) * b)
        return new * self.W, ((cur * self.W).reshape(-1)[self.ri] * self.rw).sum(1)

    def _inject(self, u, wav, scale=None):
        add = wav[:, None] * self.sw
        if scale is not None:
            add = add * scale.reshape(-1)[self.si]
        return u.reshape(-1).index_add(0, self.si.reshape(-1), add.reshape(-1)).reshape(u.shape)

    # the GPU programs' scheme
    def _init_gpu(self):
        c, nd, nb, p = self.c, self.nd, self.nb, self.p
        shell = c["coords"] != "cart"
        pri = {("cart", 2): [1, 0], ("cart", 3): [1, 2, 0], ("polar", 2): [0, 1], ("shell", 3): [0, 2, 1]}
        at = [torch.arange(p[a], device="cuda").reshape([-1] + [1] * a).expand(p[::-1]) for a in range(nd)]
        low, high = (torch.zeros(p[::-1], dtype=torch.long, device="cuda") for _ in range(2))
        for a in reversed(pri[(c["coords"], nd)]):
            low = torch.where(at[a] < nb, nb - at[a], low)
            high = torch.where(at[a] > p[a] - nb, at[a] - (p[a] - nb), high)
        i = torch.where(low > 0, low, high)
        tab = [1.0] + [math.exp(-abs((k - 1.0) ** 2 * float(np.log(np.float32(0.9)))) / nb ** 2)
                       for k in range(1, nb + 1)]
        self.W = torch.tensor(tab, **F64)[i]
        keep = torch.ones(p[::-1], dtype=torch.bool, device="cuda")
        if not shell and nd == 2:
            keep &= ~((at[1] > p[1] - nb) | ((at[1] < 8 * ((p[1] + 7) // 8) - p[1]) & (at[0] >= 1)))
        elif not shell:
            keep &= at[0] >= nb
        elif c["free"]:
            rest = at[1] >= 1
            if nd == 3:
                rest = rest | (at[2] >= 1)
            keep &= ~((at[0] > p[0] - nb) | ((at[0] < 8 * ((p[0] + 7) // 8) - p[0]) & rest))
        self.M = keep.double()
        if shell:
            f32 = np.float32
            ra = (f32(self.d[0]) * np.arange(p[0], dtype=f32) + self.opad[0]).astype(f32).astype(np.float64)
            th = (f32(self.d[1]) * np.arange(p[1], dtype=f32) + self.opad[1]).astype(f32).astype(np.float64)
            self.ra = torch.from_numpy(ra).cuda()
            self.th = torch.from_numpy(th).cuda()[:, None]
        v = self.v.reshape(-1).cpu().numpy() if not shell or nd == 2 else None
        coef = lambda q: (1 - q) / (1 + q)  # noqa: E731
        dt, nop = self.dt, 4
        self.vel2 = self.v * self.v * self.dt2
        if nd == 2:  # one-way coefficients of the last sample, the program's flat indices
            n_in, n_sw, dd = (p[1], p[0], self.d[0]) if not shell else (p[0], p[1], self.d[1])
            self.b2 = [float(coef(v[r * n_in + n_in - 1] * (dt / dd))) for r in (nop, n_sw - nop - 1)]
        elif not shell:
            nz, nx, ny = p
            t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
            V = v.reshape(ny, nz, nx)  # flat index y*n2 + z*nx + x
            k = [dt / q for q in self.d]
            self.b3 = [t(coef(V[:, nop, :] * k[0])), t(coef(V[:, nz - nop - 1, :] * k[0])),
                       t(coef(V[:, :, nop] * k[1])), None, t(coef(V[nop] * k[2])), t(coef(V[ny - nop - 1] * k[2]))]

    def _lap_gpu(self, u):
        s = lambda k, a: self._sh(u, 4, k, a)  # noqa: E731
        d2 = lambda a: s(1, a) - 2 * s(0, a) + s(-1, a)  # noqa: E731
        if self.c["coords"] == "cart":
            return sum(d2(a) / self.d[a] ** 2 for a in range(self.nd))
        ra, th = self.ra[4:-4], self.th[4:-4]
        dr, dth = self.d[0], self.d[1]
        if self.nd == 2:
            am, ap = 1 / dr ** 2 + 1 / (2 * ra * dr), 1 / dr ** 2 - 1 / (2 * ra * dr)
            return am * s(-1, 0) - 2 / dr ** 2 * s(0, 0) + ap * s(1, 0) + d2(1) / (ra ** 2 * dth ** 2)
        out = (2 / ra) * (s(1, 0) - s(-1, 0)) / (2 * dr) + d2(0) / dr ** 2
        out = out + torch.cos(th) / (ra ** 2 * torch.sin(th)) * (s(1, 1) - s(-1, 1)) / (2 * dth)
        out = out + d2(1) / dth ** 2 / ra ** 2
        return out + d2(2) / self.d[2] ** 2 / (ra ** 2 * torch.sin(th) ** 2)

    def _step_gpu(self, prv, cur, vel2, wav):
        """(levels before the injection) -> (new level, injected level, traces)."""
        cur = self._inject(cur, wav)
        new = 2 * cur - prv * self.W
        inner = tuple(slice(4, q - 4) for q in reversed(self.p))
        new[inner] = new[inner] + vel2[inner] * self._lap_gpu(cur)
        p, nd = self.p, self.nd
        if self.c["coords"] == "shell":
            new = new * self.M * self.W
        elif nd == 2:
            sw = 0 if self.c["coords"] == "cart" else 1  # swept axis; rows read at the last sample of the other
            dim, oth = (1, 0) if sw == 0 else (0, 1)
            out = new.clone()
            last = lambda x, r: x.select(dim, r)[-1]  # noqa: E731
            for k in range(8):
                r = 1 + k if k < 4 else p[sw] - 9 + k
                if sw == 0 and r >= p[1]:
                    continue
                q = r + 1 if k < 4 else r - 1
                b = self.b2[0 if k < 4 else 1]
                out.select(dim, r).copy_(last(cur, q) + (cur.select(dim, r) - last(new, q)) * b)
            new = out * self.W * self.M
        else:
            ps = new * self.M
            out = ps.clone()
            nz, nx, ny = p
            b = self.b3
            zh_of_x = b[1].reshape(-1)[(torch.arange(ny, device="cuda")[:, None] * nz
                                        + torch.arange(nz, device="cuda")[None, :])]  # [y][z], the z-high table
            one = lambda m, c_, u_, q: m + (c_ - u_) * q  # noqa: E731
            for r in range(5):
                out[..., r] = one(cur[..., r + 1], cur[..., r], ps[..., r + 1], b[0])
            for r in range(nz - 5, nz):
                m = (cur[..., r - 1], cur[..., r], ps[..., r - 1])
                out[..., r] = one(*m, b[1])
            for r in range(5):
                out[:, r] = one(cur[:, r + 1], cur[:, r], ps[:, r + 1], b[2])
            for r in range(nx - 5, nx):
                out[:, r] = one(cur[:, r - 1], cur[:, r], ps[:, r - 1], zh_of_x)
            for r in range(5):
                out[r] = one(cur[r + 1], cur[r], ps[r + 1], b[4].T)
            for r in range(ny - 5, ny):
                out[r] = one(cur[r - 1], cur[r], ps[r - 1], b[5].T)
            new = out * self.W
        return new, cur, (new.reshape(-1)[self.ri] * self.rw).sum(1)

    def _frame(self, u):
        """The model window of a level (polar: theta fastest), as the programs write it."""
        for a in range(self.nd):
            u = u.narrow(self.nd - 1 - a, self.cut[a], self.p[a] - 2 * self.nb)
        return (u.T if self.c["coords"] == "polar" else u).reshape(-1)

    def forward(self, wav, keep=False):
        """Traces [nt][nr]; with keep the two levels before every step too."""
        self.frames = []
        z = torch.zeros(self.p[::-1], **F64)
        prv, cur, rows, levels = z, z.clone(), [], []
        for it in range(self.c["nt"]):
            if keep:
                levels.append((prv, cur))
            w = wav[it].expand(self.si.shape[0])
            if self.c["program"] == "cpu":
                new, row = self._step_cpu(prv, cur, self.vel2, w)
                shown = cur * self.W
                prv, cur = cur, new
            else:
                new, done, row = self._step_gpu(prv, cur, self.vel2, w)
                prv, cur = done, new
                shown = cur
            rows.append(row)
            if self.c["snap"] and it % self.c["snap"] == 0:
                self.frames.append(self._frame(shown))
        dat = torch.stack(rows)
        if self.c["program"] == "gpu" and self.c["coords"] == "cart" and self.nd == 3:
            dat = torch.cat([torch.zeros_like(dat[:1]), dat[:-1]])  # the program's rows start at 1
        return (dat, levels) if keep else dat

    def gradient(self, wav, obs):
        """(dJ/dm on the padded grid, J), J = 0.5 ||d - obs||^2, m = 1/v^2."""
        with torch.no_grad():
            dat, levels = self.forward(wav, True)
        res = dat - obs
        lam_p = torch.zeros(self.p[::-1], **F64)
        lam_c = torch.zeros_like(lam_p)
        G = torch.zeros_like(lam_p)
        for it in reversed(range(self.c["nt"])):
            prv, cur = (q.detach().requires_grad_() for q in levels.pop())
            vel2 = self.vel2.detach().requires_grad_()
            w = wav[it].expand(self.si.shape[0])
            if self.c["program"] == "cpu":
                new, row = self._step_cpu(prv, cur, vel2, w)
                outs, gouts = [new, row, cur * 1.0], [lam_c, res[it], lam_p]
            else:
                new, done, row = self._step_gpu(prv, cur, vel2, w)
                outs, gouts = [new, row, done], [lam_c, res[it], lam_p]
            a, b, g = torch.autograd.grad(outs, [prv, cur, vel2], gouts)
            lam_p, lam_c = a, b
            G += g
        return G * (-self.vel2 ** 2 / self.dt2), 0.5 * float((res * res).sum())


def _cost(c):
    """Rough seconds of the run in 64 bits."""
    grad = c["op"].endswith("gradient")
    cells = math.prod(n + 2 * c["nb"] for n in _axes(c)[0])
    if c["op"].startswith("survey"):
        cells = _cells(c) / c["shots"]
    ops = (8 + 4 * c["order"] // 2 * _dims(c)) + (90 if _dims(c) == 3 and c["program"] == "cpu" else 20)
    step = ops * 8e-6 + cells * (8 + 2 * c["order"] * _dims(c)) * 8 / 2.5e12
    return c["nt"] * c["shots"] * step * (4 if grad else 1), cells * 8 * (2 if grad else 0) * c["nt"]


def exact(case, seed):
    c = case
    seconds, held = _cost(c)
    if seconds > 14 or held > 60e9:
        return None
    s = _inputs(c, seed)
    wav = torch.from_numpy(s["wav"]).cuda().double()
    dats, J = [], 0.0
    grad = torch.zeros(s["vel"].shape, **F64)
    for k, (x0, nx, sou, rec) in enumerate(s["shots"]):
        vel = s["vel"] if not c["op"].startswith("survey") else np.ascontiguousarray(s["vel"][x0:x0 + nx])
        g = _Grid(c, vel, s["den"], sou, rec, np.float32(np.float32(x0) * np.float32(D)) if x0 else 0.0)
        if c["op"].endswith("gradient"):
            G, j = g.gradient(wav, torch.from_numpy(s["obs"][k]).cuda().double())
            G, J = g.fold(G), J + j
            if c["op"] == "gradient":
                grad += G
            else:
                grad[x0:x0 + nx] += G
        else:
            dats.append(g.forward(wav))
    if c["op"].endswith("gradient"):
        return [grad if c["op"] == "gradient" else grad.cpu().numpy(), J]
    if c["op"] == "survey":
        return [torch.cat([q.reshape(-1) for q in dats])]
    return [torch.cat(dats, 1)] + ([torch.stack(g.frames)] if c["snap"] else [])
