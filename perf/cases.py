"""Measured workloads: the time loops, batches and gradients that users of this
framework run, each through its public Python classes.

A case is a dict of plain values; its "kind" names the path:

  steps2d    the reference drivers' loop, one update_* call per time step
  run2d      one 2D shot, the whole loop in one run()
  batch2d    many ragged 2D shots together (ShotBatch2D)
  fwi2d      one full-waveform-inversion gradient step over ragged 2D shots
  run3d      one 3D shot (moment tensor or point force; exact or fast, f32 or f64)
  spml3d     one 3D shot with the split-field PML
  grad3d     3D seismogram and the gradient of its misfit (forward_op + backward)
  learned3d  3D shot on the thin grid with the learned absorbing layer's
             correction after every step

Models, sources and observed traces are made from the seed alone.  exact()
restates each scheme in plain float64 torch on full grids.
"""
import math

import numpy as np
import torch

DEV = "cuda"
FIELDS2 = ("vx", "vz", "sxx", "szz", "sxz")
FIELDS3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")
AXES = ("x", "y", "z")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest calls: a driver script stepping a small model from Python
        # (`for i in range(nt): w.update_SSG_VS(i)`), point force, the classes'
        # default order
        dict(name="steps2d small", kind="steps2d", scheme="VS", nx=121, nz=90, order=3, h=10.0, dt=1e-3,
             freq=25.0, nt=100, mt=False, f64=False),
        # config 1: one homogeneous 400 x 400 shot, explosive source, 200 receivers
        dict(name="run2d 400", kind="run2d", scheme="VS", nx=400, nz=400, order=2, h=10.0, dt=1e-3, freq=25.0,
             nt=1000, nrec=200, model="homogeneous", src="centre", mt=True, f64=False),
        # config 4's batch: ragged heterogeneous shots, (nx, nz) in 600-1200 x 300-500
        dict(name="batch2d ragged", kind="batch2d", scheme="VS", nshots=32, nx0=600, nx1=1200, nz0=300, nz1=500,
             shapes=4, order=2, h=10.0, dt=1e-3, freq=15.0, nt=200),
        # config 4's gradient step on a part of its shots; the last checkpoint
        # interval is shorter than the others
        dict(name="fwi2d ragged", kind="fwi2d", nshots=8, nx0=600, nx1=1200, nz0=300, nz1=500, shapes=4, order=2,
             h=10.0, dt=1e-3, freq=15.0, nt=240, every=100),
        # config 2: the 3D forward run of the benchmark, 200^3, double couple
        dict(name="run3d 200", kind="run3d", source="tensor", nx=200, ny=200, nz=200, order=2, h=10.0, dt=1e-3,
             freq=15.0, nt=600, nrec=50, npml=20, model="homogeneous", src="centre", exact=True, f64=False),
        # config 3's grid: the largest, heterogeneous
        dict(name="run3d thrust", kind="run3d", source="tensor", nx=400, ny=400, nz=200, order=2, h=12.5, dt=8e-4,
             freq=10.0, nt=150, nrec=50, npml=20, model="layered", exact=True, f64=False),
        # the faster numeric mode on a higher-order grid
        dict(name="run3d fast", kind="run3d", source="tensor", nx=240, ny=180, nz=160, order=4, h=10.0, dt=8e-4,
             freq=15.0, nt=200, nrec=30, npml=20, model="layered", exact=False, f64=False),
        # a model whose sides come from the survey, not from a tile: odd sides,
        # point force
        dict(name="run3d odd", kind="run3d", source="force", nx=153, ny=131, nz=117, order=3, h=10.0, dt=8e-4,
             freq=15.0, nt=200, nrec=1, npml=20, model="layered", exact=True, f64=False),
        # double precision, as used to judge the single-precision runs
        dict(name="run3d f64", kind="run3d", source="tensor", nx=128, ny=120, nz=112, order=2, h=10.0, dt=1e-3,
             freq=15.0, nt=150, nrec=20, npml=20, model="layered", exact=True, f64=True),
        # the split-field PML scheme at the benchmark's grid
        dict(name="spml3d 200", kind="spml3d", nx=200, ny=200, nz=200, order=2, h=10.0, dt=1e-3, freq=15.0, nt=200,
             npml=20, model="homogeneous"),
        # the gradient of a 3D misfit with respect to vp, vs and rho
        dict(name="grad3d", kind="grad3d", nx=104, ny=96, nz=80, order=2, h=10.0, dt=1e-3, freq=15.0, nt=130,
             nrec=20, npml=10, every=100),
        # config 5's learned layer on a smaller interior
        dict(name="learned3d", kind="learned3d", nx=144, ny=144, nz=144, order=2, h=10.0, dt=1e-3, freq=12.0, nt=60,
             nrec=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps2d", "run2d", "run2d", "batch2d", "fwi2d", "run3d", "run3d", "run3d", "run3d", "spml3d",
                       "grad3d", "learned3d"])
    h = rng.choice([5.0, 8.0, 10.0, 12.5])
    order = rng.choice([1, 2, 2, 2, 3, 3, 4])
    # h*dt keep a Courant number near 0.42 (2D) / 0.52 (3D) for vp <= 4500 m/s
    c = dict(kind=kind, order=order, h=h, dt=round(9e-5 * h, 7), freq=round(rng.uniform(0.08, 0.16) * 1500.0 / h, 1))
    if kind == "steps2d":
        c.update(scheme=rng.choice(["VS", "SV"]), nx=rng.randint(60, 320), nz=rng.randint(60, 320),
                 nt=rng.randint(40, 120), mt=rng.random() < 0.5, f64=rng.random() < 0.2)
    elif kind == "run2d":
        c.update(scheme=rng.choice(["VS", "VS", "SV"]), nx=_log(rng, 100, 1400), nz=_log(rng, 100, 900),
                 nt=rng.randint(200, 800), nrec=rng.randint(1, 200), model=rng.choice(["homogeneous", "layered"]),
                 mt=rng.random() < 0.7, f64=rng.random() < 0.2)
    elif kind in ("batch2d", "fwi2d"):
        fwi = kind == "fwi2d"
        nx0, nz0 = rng.randint(150, 700), rng.randint(120, 350)
        c.update(nshots=rng.randint(2, 8) if fwi else rng.randint(4, 40), nx0=nx0, nx1=nx0 + rng.randint(20, 500),
                 nz0=nz0, nz1=nz0 + rng.randint(20, 200), shapes=rng.randint(2, 4), nt=rng.randint(120, 240))
        c.update({"every": rng.choice([50, 100])} if fwi else {"scheme": rng.choice(["VS", "SV"])})
    elif kind == "run3d":
        f64 = rng.random() < 0.25
        n = [_log(rng, 60, 260) for _ in range(3)]
        if rng.random() < 0.5:
            n[2] = max(60, n[2] // 4 * 4)
        cells = n[0] * n[1] * n[2]
        c.update(source=rng.choice(["tensor", "force"]), nx=n[0], ny=n[1], nz=n[2],
                 nt=min(300, max(30, int(4e8 / cells))), nrec=rng.randint(1, 40), npml=rng.choice([10, 20]),
                 model=rng.choice(["homogeneous", "layered"]), exact=f64 or rng.random() < 0.7, f64=f64)
    elif kind == "spml3d":
        n = [_log(rng, 60, 220) for _ in range(3)]
        if rng.random() < 0.7:
            n[2] = max(60, n[2] // 4 * 4)
        c.update(nx=n[0], ny=n[1], nz=n[2], nt=min(200, max(30, int(3e8 / (n[0] * n[1] * n[2])))),
                 npml=rng.choice([10, 20]), model=rng.choice(["homogeneous", "layered"]))
    elif kind == "grad3d":
        c.update(nx=rng.randint(50, 110), ny=rng.randint(50, 110), nz=rng.randint(50, 90), nt=rng.randint(60, 130),
                 nrec=rng.randint(4, 30), npml=10, every=rng.choice([40, 100]))
    else:
        c.update(order=2, nx=rng.randint(64, 150), ny=rng.randint(64, 150), nz=rng.randint(16, 37) * 4,
                 nt=rng.randint(30, 60), nrec=rng.randint(4, 30))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _f64(case):
    return bool(case.get("f64"))


def _dtype(case):
    return torch.float64 if _f64(case) else torch.float32


def _model(shape, kind, seed):
    """vp, vs, rho (float32, on the GPU): one value, or layers along the last
    axis with a smooth lateral perturbation, 2000-4500 m/s, vs = vp/1.73,
    Gardner density."""
    r = np.random.default_rng(seed)
    if kind == "homogeneous":
        vp = torch.full(shape, float(r.uniform(2900, 3100)), device=DEV)
        return vp, vp / 1.732, torch.full(shape, float(r.uniform(1900, 2100)), device=DEV)
    n = len(shape)
    nz = shape[-1]
    cut = np.sort(r.uniform(0.1, 0.9, 7)) * nz
    lay = torch.as_tensor(np.searchsorted(cut, np.arange(nz)), device=DEV, dtype=torch.float32)
    vp = 2000.0 + 2200.0 / 7 * lay
    vp = vp.reshape([1] * (n - 1) + [nz]).expand(shape).clone()
    for a in range(n):
        ph, w = r.uniform(0, 2 * math.pi), r.integers(1, 4)
        s = torch.sin(2 * math.pi * float(w) * torch.arange(shape[a], device=DEV) / shape[a] + ph)
        vp *= 1 + 0.02 * s.reshape([-1 if q == a else 1 for q in range(n)])
    return vp, vp / 1.73, 1741.0 * (vp / 1000.0) ** 0.25


def _pml(case, vp, vs, npml, dims):
    h, f = case["h"], case["freq"]
    p = {"vp_max": float(vp.max()), "Rcoef": 1e-6, "theta": 1, "alpha_max_pml": math.pi * f,
         "kmax_pml": max(1.0, float(vs.max()) / (5 * h * f))}
    for ax in ("xyz" if dims == 3 else "xz"):
        p["pml_%s_thick" % ax] = npml * h
    return p


def _source(case, r, shape):
    """Source cell within a tenth of the middle; its depth (the last axis) 8 to
    24 cells below the top of the PML-free grid unless the case says centre."""
    at = [int(n // 2 + r.integers(-n // 10, n // 10 + 1)) for n in shape]
    shallow = min(shape[-1] // 2, case["order"] + int(r.integers(8, 25)))
    return at if case.get("src") == "centre" else at[:-1] + [shallow]


def _inputs2(case, seed, nx, nz):
    r = np.random.default_rng(seed + 7)
    N = case["order"]
    vp, vs, rho = _model((nx, nz), case.get("model", "layered"), seed)
    nrec = case.get("nrec") or max(2, (nx - 2 * N - 42) // 4)
    rx = np.linspace(N + 2, nx - N - 3, nrec).astype(np.int64).reshape(1, -1)
    rz = np.full_like(rx, N + 5)
    isx, isz = _source(case, r, (nx, nz))
    return dict(vp=vp, vs=vs, rho=rho, isx=isx, isz=isz, rsx=rx, rsz=rz, pml=_pml(case, vp, vs, 20, 2))


def _scale2(case):
    return 1e6 if case["kind"] == "fwi2d" else 1.0


def _wave2(case, d, mt):
    from seiswave_taichi_b200.Elastic2D_CPML import ElasticWAVE
    w = ElasticWAVE(d["vs"], d["vp"], d["rho"], case["h"], case["h"], case["dt"], d["isx"], d["isz"], d["rsx"],
                    d["rsz"], case["nt"], case["order"], case["freq"], _dtype(case), MT="explosive" if mt else None,
                    src_scale=_scale2(case))
    w.SetADEPML2D([True] * 4, d["pml"])
    return w


def _inputs3(case, seed):
    r = np.random.default_rng(seed + 7)
    N = case["order"]
    shape = (case["nx"], case["ny"], case["nz"])
    npml = case.get("npml", 6)
    vp, vs, rho = _model(shape, case.get("model", "layered"), seed)
    m = r.standard_normal(6)
    M = np.array([[m[0], m[3], m[4]], [m[3], m[1], m[5]], [m[4], m[5], m[2]]], np.float32)
    g = case.get("nrec", 1)
    X, Y = np.meshgrid(np.linspace(N + 8, shape[0] - N - 9, g).astype(np.int64),
                       np.linspace(N + 8, shape[1] - N - 9, g).astype(np.int64), indexing="ij")
    src = _source(case, r, shape)
    if case["kind"] == "spml3d" or case.get("source") == "force":  # one receiver, beside the shot
        rec = [np.array([[src[0] - 6]]), np.array([[src[1] + 4]]), np.array([[N + 5]])]
    else:
        rec = [X.reshape(1, -1), Y.reshape(1, -1), np.full((1, g * g), N + 5, np.int64)]
    return dict(vp=vp, vs=vs, rho=rho, src=src, rec=rec, MT=M, pml=_pml(case, vp, vs, npml, 3))


def _wave3(case, d):
    if case["kind"] == "spml3d":
        from seiswave_taichi_b200.Elastic3D_SSG_SPML import ElasticWAVE
    elif case.get("source") == "force":
        from seiswave_taichi_b200.Elastic3D_SSG_CPML import ElasticWAVE
    else:
        from seiswave_taichi_b200.Elastic3D_SSG_Tensor import ElasticWAVE
    h = case["h"]
    a = [d["vs"], d["vp"], d["rho"], h, h, h, case["dt"], *d["src"]]
    rec = [int(q[0, 0]) for q in d["rec"]]
    if case["kind"] == "spml3d":
        w = ElasticWAVE(*a, *rec, case["nt"], case["order"], case["freq"], 1000.0)
    elif case.get("source") == "force":
        w = ElasticWAVE(*a, *rec, case["nt"], case["order"], case["freq"], _dtype(case), exact=case["exact"])
    else:
        w = ElasticWAVE(*a, *d["rec"], d["MT"], 1e6, case["nt"], case["order"], case["freq"], _dtype(case),
                        exact=case.get("exact", True))
    w.SetADEPML3D([True] * 6, d["pml"])
    return w


def _shots(case, seed):
    """Ragged shots: `shapes` distinct grids used in turn, every shot its own
    model, source and receivers."""
    r = np.random.default_rng(12345)
    shapes = [(int(r.integers(case["nx0"], case["nx1"] + 1)), int(r.integers(case["nz0"], case["nz1"] + 1)))
              for _ in range(case["shapes"])]
    return [_inputs2(case, 1000 * seed + s, *shapes[s % len(shapes)]) for s in range(case["nshots"])]


def _observed(case, d, seed):
    """Observed traces: one hyperbolic arrival with noise."""
    nt, dt, f = case["nt"], case["dt"], case["freq"]
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    x = torch.as_tensor((d["rsx"][0] - d["isx"]) * case["h"], device=DEV, dtype=torch.float32)
    z = float(d["rsz"][0, 0] - d["isz"]) * case["h"]
    t = torch.arange(nt, device=DEV, dtype=torch.float32)[:, None] * dt
    a = (math.pi * f * (t - 1.0 / f - torch.sqrt(x * x + z * z)[None, :] / 3000.0)) ** 2
    noise = torch.randn((nt, x.numel()), generator=g, device=DEV)
    return 1e-2 * ((1 - 2 * a) * torch.exp(-a) + 0.02 * noise)


def _net(case, seed):
    """Six faces' networks as a trained layer has them: Glorot hidden layers,
    a small output layer."""
    r = np.random.default_rng(seed + 99)
    NI, NH, NO = 33, 32, 9
    rows = []
    for _ in range(6):
        rows.append(np.concatenate([
            (r.uniform(-1, 1, (NH, NI)) * math.sqrt(6.0 / (NI + NH))).reshape(-1), 0.1 * r.standard_normal(NH),
            (r.uniform(-1, 1, (NH, NH)) * math.sqrt(6.0 / (2 * NH))).reshape(-1), 0.1 * r.standard_normal(NH),
            (0.1 * r.standard_normal((NO, NH))).reshape(-1), 0.01 * r.standard_normal(NO)]))
    scale = np.array([1e-2] * 3 + [5e4] * 6)
    return np.stack(rows).astype(np.float32), scale.tolist(), (1e-4 * scale).tolist()


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    k = case["kind"]
    if k in ("steps2d", "run2d"):
        return dict(case=case, w=_wave2(case, _inputs2(case, seed, case["nx"], case["nz"]), case["mt"]))
    if k == "batch2d":
        from seiswave_taichi_b200.batch import ShotBatch2D
        waves = [_wave2(case, d, True) for d in _shots(case, seed)]
        return dict(case=case, b=ShotBatch2D(waves, case["scheme"]), waves=waves)
    if k == "fwi2d":
        from seiswave_taichi_b200.fwi import FWIStep
        shots = _shots(case, seed)
        waves = [_wave2(case, d, True) for d in shots]
        obs = [_observed(case, d, 1000 * seed + s) for s, d in enumerate(shots)]
        return dict(case=case, step=FWIStep(waves, checkpoint_every=case["every"]), obs=obs)
    d = _inputs3(case, seed)
    if k == "learned3d":
        from seiswave_taichi_b200.learned_abc3d import LearnedABC3D
        return dict(case=case, w=_wave3(case, d), abc=LearnedABC3D(*_net(case, seed)))
    w = _wave3(case, d)
    if k == "grad3d":
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        res = torch.randn((case["nt"], int(w.datasize)), generator=g, device=DEV)
        return dict(case=case, w=w, m=[d[q] for q in ("vp", "vs", "rho")], res=res)
    return dict(case=case, w=w)


def run(state):
    case, w = state["case"], state.get("w")
    k, nt = case["kind"], case["nt"]
    if k == "steps2d":
        w.reset()
        step = w.update_SSG_VS if case["scheme"] == "VS" else w.update_SSG_SV
        for i in range(nt):
            step(i)
        return [w.data] + [getattr(w, f) for f in FIELDS2]
    if k == "run2d":
        w.reset()
        w.run(nt, scheme=case["scheme"])
        return [w.data] + [getattr(w, f) for f in FIELDS2]
    if k == "batch2d":
        state["b"].reset()
        state["b"].run()
        last = state["waves"][-1]
        return [x.data for x in state["waves"]] + [getattr(last, f) for f in FIELDS2]
    if k == "fwi2d":
        misfit, grads = state["step"](state["obs"])
        return [misfit] + [list(g) for g in grads]
    if k == "grad3d":
        m = [t.detach().clone().requires_grad_(True) for t in state["m"]]
        d = w.forward_op(*m, checkpoint_every=case["every"])
        d.backward(state["res"])
        return [d.detach()] + [t.grad for t in m]
    w.reset()
    if k == "learned3d":
        state["abc"].run(w, nt)
    else:
        w.run(nt)
    return [w.data] + [getattr(w, f) for f in FIELDS3]


# ---------------------------------------------------------------------------
# the least work of a pass: per time step every wavefield and memory variable
# (split field) read and written once and every material read once
# ---------------------------------------------------------------------------
def _slab(n, npml):
    """Cells of all axes' PML slabs, counted per axis."""
    tot = math.prod(n)
    return sum(min(a, 2 * npml + 2) * (tot // a) for a in n)


def _work2(case, nx, nz):
    cells, e = nx * nz, 8 if _f64(case) else 4
    return cells * 13 * e + _slab((nx, nz), 20) * 8 * e, cells * (8 * 3 * case["order"] + 40)


def work(case):
    k, nt, N = case["kind"], case["nt"], case["order"]
    if k in ("steps2d", "run2d"):
        b, f = _work2(case, case["nx"], case["nz"])
        return dict(bytes=b * nt, flops=f * nt)
    if k in ("batch2d", "fwi2d"):
        nx, nz = (case["nx0"] + case["nx1"]) // 2, (case["nz0"] + case["nz1"]) // 2
        b, f = _work2(case, nx, nz)
        b, f = b * nt * case["nshots"], f * nt * case["nshots"]
        if k == "fwi2d":  # the forward, its replay, and the adjoint (own state twice, forward state, gradients)
            cells = nx * nz * nt * case["nshots"]
            b, f = 2 * b + cells * 4 * (10 + 5 + 3 + 10), 4 * f
        return dict(bytes=b, flops=f)
    n = (case["nx"], case["ny"], case["nz"])
    cells, e = math.prod(n), 8 if _f64(case) else 4
    npml = case.get("npml", 6)
    flops = cells * (18 * 3 * N + 100)
    if k == "spml3d":
        shell = cells - math.prod(max(0, a - 2 * npml - 2) for a in n)
        return dict(bytes=nt * (cells * 84 + shell * 192), flops=nt * flops)
    b = cells * 21 * e + _slab(n, npml) * 12 * e
    if k == "grad3d":
        return dict(bytes=nt * (2 * b + cells * 4 * (18 + 9 + 3 + 16) + _slab(n, npml) * 72), flops=nt * 4 * flops)
    if k == "learned3d":
        layer = cells - math.prod(a - 12 for a in n)
        return dict(bytes=nt * (b + layer * 9 * 8), flops=nt * (flops + layer * 2 * (33 * 32 + 32 * 32 + 9 * 32)))
    return dict(bytes=nt * b, flops=nt * flops)


# ---------------------------------------------------------------------------
# float64 restatement
# ---------------------------------------------------------------------------
def _coef(N):
    A = np.array([[(2 * j + 1) ** (2 * i + 1) for j in range(N)] for i in range(N)], float)
    b = np.zeros(N)
    b[0] = 1
    return [float(np.float32(v)) for v in np.linalg.solve(A, b)]  # the scheme's coefficients are stored in float32


def _ricker(nt, dt, f, s):
    t = np.arange(nt) * dt - 1.5 / f
    a = math.pi ** 2 * f * f
    return (-s * 2 * a * t * np.exp(-a * t * t)).tolist()


def _ricker2(nt, dt, t0, f, s):
    t = np.arange(nt) * dt - t0
    a = math.pi ** 2 * f * f
    return (s * (1 - 2 * a * t * t) * np.exp(-a * t * t)).tolist()


class _Axis:
    """One axis' PML profiles at integer (0) and half (1) points, and where the
    PML predicate holds."""

    def __init__(self, n, N, h, p, dt, thick):
        lo, hi = thick, h * (n - 1 - 2 * N) - thick
        d0 = -3.0 * p["vp_max"] * math.log(p["Rcoef"]) / (2.0 * thick)
        self.b, self.a, self.k, self.d, self.on = [], [], [], [], []
        for half in (0, 1):
            x = (np.arange(n) - N) * h + half * h / 2
            s = np.where(x <= lo, (lo - x) / thick, np.where(x >= hi, (x - hi) / thick, 0.0))
            inside = (x <= lo) | (x >= hi)
            d = d0 * s ** 2 * inside
            al = np.maximum(p["alpha_max_pml"] * (1 - s) * inside, 0.0)
            k = np.where(inside, 1 + (p["kmax_pml"] - 1) * s ** 2, 1.0)
            den = 1 + dt * (d / k + al)
            self.b.append(1 / den)
            self.a.append(np.where(np.abs(d) > 1e-6, -dt * d / (k * k) / den, 0.0))
            self.k.append(k)
            self.d.append(d)
            self.on.append(inside)


class _Scheme:
    """Full-grid float64 state and the difference and CPML operators on it."""

    def __init__(self, case, shape, pml, dims):
        self.shape, self.N, self.h, self.dt = shape, case["order"], case["h"], case["dt"]
        self.c = [v / self.h for v in _coef(self.N)]
        names = "xz" if dims == 2 else "xyz"
        self.ax = [_Axis(n, self.N, self.h, pml, self.dt, pml["pml_%s_thick" % a]) for n, a in zip(shape, names)]
        self.psi, self.tab = {}, {}

    def zeros(self):
        return torch.zeros(self.shape, dtype=torch.float64, device=DEV)

    def win(self, w):
        return tuple(slice(a, b) for a, b in w)

    def at(self, f, w, **shift):
        """f on window w, moved by shift["a0"|"a1"|"a2"] cells."""
        return f[tuple(slice(a + shift.get("a%d" % q, 0), b + shift.get("a%d" % q, 0)) for q, (a, b) in enumerate(w))]

    def vec(self, what, axis, half, w):
        key = (what, axis, half, w[axis])
        if key not in self.tab:
            v = getattr(self.ax[axis], what)[half][w[axis][0]:w[axis][1]]
            self.tab[key] = torch.as_tensor(v, device=DEV).reshape([-1 if q == axis else 1 for q in range(len(w))])
        return self.tab[key]

    def raw(self, f, axis, fwd, w):
        out, a = None, "a%d" % axis
        for m, c in enumerate(self.c):
            hi, lo = (m + 1, -m) if fwd else (m, -m - 1)
            t = (self.at(f, w, **{a: hi}) - self.at(f, w, **{a: lo})) * c
            out = t if out is None else out + t
        return out

    def d(self, f, axis, fwd, w, half, name):
        """CPML-corrected derivative; memory variable `name`, profiles at the
        half points of the axis where half is set."""
        v = self.raw(f, axis, fwd, w)
        key = (name, axis)
        if key not in self.psi:
            self.psi[key] = torch.zeros_like(v)
        p = self.vec("b", axis, half, w) * self.psi[key] + self.vec("a", axis, half, w) * v
        self.psi[key] = p
        return v / self.vec("k", axis, half, w) + p


def _add(f, w, inc):
    f[tuple(slice(a, b) for a, b in w)] += inc


def _sim2(case, d, scheme, mt, model=None):
    """(traces, five fields) of one 2D shot."""
    nx, nz = d["vp"].shape
    N, dt, f = case["order"], case["dt"], case["freq"]
    vp, vs, rho = model or [d[q].to(_dtype(case)).double() for q in ("vp", "vs", "rho")]
    mu, lam = rho * vs * vs, rho * (vp * vp - 2 * vs * vs)
    S = _Scheme(case, (nx, nz), d["pml"], 2)
    vx, vz, sxx, szz, sxz = (S.zeros() for _ in range(5))
    wav = _ricker2(case["nt"], dt, float(np.float32(1.5 / f)), f, _scale2(case)) if scheme == "VS" else \
        _ricker(case["nt"], dt, f, _scale2(case))
    I, B = lambda n: (N + 1, n - N), lambda n: (N, n - N - 1)
    if scheme == "VS":
        wx, wz, wn, ws = (I(nx), I(nz)), (B(nx), B(nz)), (B(nx), I(nz)), (I(nx), B(nz))
        rx = S.at(rho, wx)
        rz = 0.25 * (S.at(rho, wz) + S.at(rho, wz, a1=1) + S.at(rho, wz, a0=1, a1=1) + S.at(rho, wz, a0=1))
        l, m = 0.5 * (S.at(lam, wn) + S.at(lam, wn, a0=1)), 0.5 * (S.at(mu, wn) + S.at(mu, wn, a0=1))
        ms = 0.5 * (S.at(mu, ws) + S.at(mu, ws, a1=1))
    else:
        wx, wz, wn, ws = (B(nx), I(nz)), (I(nx), B(nz)), (I(nx), I(nz)), (I(nx), I(nz))
        rx, rz = 0.5 * (S.at(rho, wx) + S.at(rho, wx, a0=1)), 0.5 * (S.at(rho, wz) + S.at(rho, wz, a1=1))
        l, m = S.at(lam, wn), S.at(mu, wn)
        ms = 0.25 * (S.at(mu, ws) + S.at(mu, ws, a1=1) + S.at(mu, ws, a0=1, a1=1) + S.at(mu, ws, a0=1))
    sv = scheme == "SV"
    si, sk = d["isx"], d["isz"]
    lin = torch.as_tensor(d["rsx"][0] * nz + d["rsz"][0], device=DEV)
    out = []
    for it in range(case["nt"]):
        if mt:
            sxx[si, sk] -= wav[it]
            szz[si, sk] -= wav[it]
        ax = S.d(sxx, 0, sv, wx, int(sv), "a") + S.d(sxz, 1, False, wx, 0, "a")
        az = S.d(sxz, 0, not sv, wz, int(not sv), "b") + S.d(szz, 1, True, wz, 1, "b")
        _add(vx, wx, ax * dt / rx)
        _add(vz, wz, az * dt / rz)
        if not mt:
            (vx if sv else vz)[si, sk] += dt * wav[it] / rho[si, sk]
        p, q = S.d(vx, 0, not sv, wn, int(not sv), "c"), S.d(vz, 1, False, wn, 0, "c")
        sh = S.d(vz, 0, sv, ws, int(sv), "e") + S.d(vx, 1, True, ws, 1, "e")
        _add(sxx, wn, ((l + 2 * m) * p + l * q) * dt)
        _add(szz, wn, ((l + 2 * m) * q + l * p) * dt)
        _add(sxz, ws, ms * sh * dt)
        out.append((vx if sv else vz).reshape(-1)[lin])
    return torch.stack(out), [vx, vz, sxx, szz, sxz]


def _windows3(nx, ny, nz, N):
    I, B, F = lambda n: (N + 1, n - N), lambda n: (N, n - N - 1), lambda n: (N, n - N)
    return dict(vx=(B(nx), I(ny), I(nz)), vy=(I(nx), B(ny), I(nz)), vz=(I(nx), I(ny), B(nz)),
                n=(I(nx), I(ny), I(nz)), xy=(I(nx), I(ny), F(nz)), xz=(B(nx), F(ny), B(nz)), yz=(F(nx), B(ny), B(nz)))


def _materials3(S, W, rho, lam, mu, spml):
    at = S.at
    r = dict(vx=at(rho, W["vx"]), vy=0.5 * (at(rho, W["vy"]) + at(rho, W["vy"], a1=1)),
             vz=0.25 * (at(rho, W["vz"]) + at(rho, W["vz"], a1=1) + at(rho, W["vz"], a0=1, a1=1) +
                        at(rho, W["vz"], a0=1)))
    n = W["n"]
    l, m = at(lam, n), at(mu, n)
    if not spml:
        l, m = 0.5 * (l + at(lam, n, a0=1)), 0.5 * (m + at(mu, n, a0=1))
    g = dict(xy=0.25 * (at(mu, W["xy"], a1=1) + 2 * at(mu, W["xy"]) + at(mu, W["xy"], a0=1)),
             xz=0.25 * (2 * at(mu, W["xz"]) + at(mu, W["xz"], a0=1) + at(mu, W["xz"], a1=1)),
             yz=0.25 * (at(mu, W["yz"], a1=1) + 2 * at(mu, W["yz"]) + at(mu, W["yz"], a2=1)))
    return r, l, m, g


def _sim3(case, d, model=None, after=None):
    """(traces, nine fields) of one 3D CPML shot; after(fields) runs after
    every step."""
    shape = nx, ny, nz = tuple(d["vp"].shape)
    N, dt, f, nt = case["order"], case["dt"], case["freq"], case["nt"]
    vp, vs, rho = model or [d[q].to(_dtype(case)).double() for q in ("vp", "vs", "rho")]
    mu, lam = rho * vs * vs, rho * (vp * vp - 2 * vs * vs)
    S = _Scheme(case, shape, d["pml"], 3)
    W = _windows3(nx, ny, nz, N)
    r, l, m, g = _materials3(S, W, rho, lam, mu, False)
    F = {q: S.zeros() for q in FIELDS3}
    force = case.get("source") == "force"
    wav = _ricker(nt, dt, f, 1000.0) if force else _ricker2(nt, dt, 0.03, f, 1e6)
    si, sj, sk = [q + 5 for q in d["src"]] if force else d["src"]
    M = d["MT"].astype(float)
    lin = torch.as_tensor((d["rec"][0][0] * ny + d["rec"][1][0]) * nz + d["rec"][2][0], device=DEV)
    out = []
    for it in range(nt):
        if not force:
            for q, (a, b) in zip(FIELDS3[3:], ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
                F[q][si, sj, sk] -= wav[it] * M[a, b]
        w = W["vx"]
        _add(F["vx"], w, (S.d(F["sxx"], 0, True, w, 1, "vx") + S.d(F["sxz"], 2, False, w, 0, "vx") +
                          S.d(F["sxy"], 1, False, w, 0, "vx")) * dt / r["vx"])
        w = W["vy"]
        _add(F["vy"], w, (S.d(F["sxy"], 0, False, w, 0, "vy") + S.d(F["syy"], 1, True, w, 1, "vy") +
                          S.d(F["syz"], 2, False, w, 0, "vy")) * dt / r["vy"])
        w = W["vz"]
        _add(F["vz"], w, (S.d(F["sxz"], 0, False, w, 0, "vz") + S.d(F["syz"], 1, False, w, 0, "vz") +
                          S.d(F["szz"], 2, True, w, 1, "vz")) * dt / r["vz"])
        if force:
            F["vz"][si, sj, sk] += dt * wav[it] / rho[si, sj, sk]
        w = W["n"]
        a, b, c = (S.d(F[q], x, False, w, 0, "n") for x, q in enumerate(("vx", "vy", "vz")))
        _add(F["sxx"], w, ((l + 2 * m) * a + l * (b + c)) * dt)
        _add(F["syy"], w, ((l + 2 * m) * b + l * (a + c)) * dt)
        _add(F["szz"], w, ((l + 2 * m) * c + l * (a + b)) * dt)
        for q, p1, a1, p2, a2 in (("xy", "vx", 1, "vy", 0), ("xz", "vx", 2, "vz", 0), ("yz", "vy", 2, "vz", 1)):
            w = W[q]
            _add(F["s" + q], w, g[q] * (S.d(F[p1], a1, True, w, 1, q) + S.d(F[p2], a2, True, w, 1, q)) * dt)
        out.append(F["vx"].reshape(-1)[lin])
        if after:
            after(F)
    return torch.stack(out), [F[q] for q in FIELDS3]


def _sim_spml(case, d):
    shape = nx, ny, nz = tuple(d["vp"].shape)
    N, dt, nt = case["order"], case["dt"], case["nt"]
    vp, vs, rho = (d[q].double() for q in ("vp", "vs", "rho"))
    mu, lam = rho * vs * vs, rho * (vp * vp - 2 * vs * vs)
    S = _Scheme(case, shape, d["pml"], 3)
    W = _windows3(nx, ny, nz, N)
    r, l, m, g = _materials3(S, W, rho, lam, mu, True)
    F = {q: S.zeros() for q in FIELDS3}
    wav = _ricker(nt, dt, case["freq"], 1000.0)
    split, mask = {}, {}

    def update(name, w, half, terms):
        """terms: {axis: rate}; half[axis]: the component's half points"""
        sl = tuple(slice(a, b) for a, b in w)
        if name not in mask:
            on = torch.zeros([b - a for a, b in w], dtype=torch.bool, device=DEV)
            for a in range(3):
                v = torch.as_tensor(S.ax[a].on[half[a]][w[a][0]:w[a][1]], device=DEV)
                on |= v.reshape([-1 if q == a else 1 for q in range(3)])
            mask[name] = on
            for a in terms:
                split[name, a] = torch.zeros(on.shape, dtype=torch.float64, device=DEV)
        tot, plain = 0, 0
        for a, t in terms.items():
            dm = S.vec("d", a, half[a], w) * (dt / 2)
            split[name, a] = torch.where(mask[name], ((1 - dm) * split[name, a] + dt * t) / (1 + dm), split[name, a])
            tot = tot + split[name, a]
            plain = plain + t
        F[name][sl] = torch.where(mask[name], tot, F[name][sl] + dt * plain)

    lin = (int(d["rec"][0][0, 0]), int(d["rec"][1][0, 0]), int(d["rec"][2][0, 0]))
    si, sj, sk = d["src"]
    out = []
    for it in range(nt):
        for q, half, parts in (("vx", (1, 0, 0), ("sxx", "sxy", "sxz")), ("vy", (0, 1, 0), ("sxy", "syy", "syz")),
                               ("vz", (0, 0, 1), ("sxz", "syz", "szz"))):
            w = W[q]
            update(q, w, half, {a: S.raw(F[p], a, bool(half[a]), w) / r[q] for a, p in enumerate(parts)})
        F["vz"][si, sj, sk] += dt * wav[it] / rho[si, sj, sk]
        w = W["n"]
        e = [S.raw(F[q], a, False, w) for a, q in enumerate(("vx", "vy", "vz"))]
        for a, q in enumerate(("sxx", "syy", "szz")):
            update(q, w, (0, 0, 0), {b: ((l + 2 * m) if a == b else l) * e[b] for b in range(3)})
        for q, half, p1, a1, p2, a2 in (("xy", (1, 1, 0), "vx", 1, "vy", 0), ("xz", (1, 0, 1), "vx", 2, "vz", 0),
                                        ("yz", (0, 1, 1), "vy", 2, "vz", 1)):
            w = W[q]
            update("s" + q, w, half, {a1: g[q] * S.raw(F[p1], a1, True, w), a2: g[q] * S.raw(F[p2], a2, True, w)})
        out.append(F["vx"][lin].clone())
    return torch.stack(out), [F[q] for q in FIELDS3]


def _layer(case, params, scale, oscale):
    """The learned layer's correction of the nine fields' outer six cells."""
    shape = (case["nx"], case["ny"], case["nz"])
    idx = torch.meshgrid(*[torch.arange(n, device=DEV) for n in shape], indexing="ij")
    dist = torch.stack([v for q, n in enumerate(shape) for v in (idx[q], n - 1 - idx[q])])
    dep, face = dist.min(dim=0)  # the first of equal faces
    strides = (shape[1] * shape[2], shape[2], 1)
    P = torch.as_tensor(params, device=DEV).double()
    sc, osc = (torch.tensor(np.float32(v), device=DEV).double() for v in (scale, oscale))
    lin = torch.arange(math.prod(shape), device=DEV).reshape(shape)
    faces = []
    for f in range(6):
        first = torch.ones_like(dep, dtype=torch.bool)
        for q in range(f):
            first &= dist[q] != dep
        sel = (dep < 6) & (dist[f] == dep) & first
        c = lin[sel]
        step = strides[f // 2] * (1 if f % 2 == 0 else -1)
        hot = torch.nn.functional.one_hot(dep[sel], 6).double()
        p, o, wb = P[f], 0, []
        for rows, cols in ((32, 33), (32, 32), (9, 32)):
            wb.append((p[o:o + rows * cols].reshape(rows, cols), p[o + rows * cols:o + rows * cols + rows]))
            o += rows * cols + rows
        faces.append((c, step, hot, wb, dep[sel]))

    def after(F):
        flat = [F[q].reshape(-1) for q in FIELDS3]
        done = []
        for c, step, hot, wb, dp in faces:
            x = _features(flat, c, step, hot, dp, sc)
            for W, b in wb[:2]:
                x = torch.tanh(x @ W.T + b)
            done.append((c, (x @ wb[2][0].T + wb[2][1]) * osc))
        for c, y in done:
            for q in range(9):
                flat[q][c] += y[:, q]
    return after


def _features(flat, c, step, hot, dep, sc):
    """Field values at the cell and its two neighbours along the inward normal
    (outward one, cell, inward one; clamped at the edge), scaled, and the
    depth."""
    cols = []
    for q in range(9):
        for s in (-1, 0, 1):
            at = torch.where(dep + s < 0, c, c + s * step)
            cols.append(flat[q][at] / sc[q])
    return torch.cat([torch.stack(cols, 1), hot], 1)


def exact(case, seed):
    k = case["kind"]
    if k in ("steps2d", "run2d"):
        t, fields = _sim2(case, _inputs2(case, seed, case["nx"], case["nz"]), case["scheme"], case["mt"])
        return [t] + fields
    if k == "batch2d":
        if case["nshots"] * case["nt"] > 8000:
            return None
        got = [_sim2(case, d, case["scheme"], True) for d in _shots(case, seed)]
        return [t for t, _ in got] + got[-1][1]
    if k == "fwi2d":
        total, grads = 0.0, []
        for s, d in enumerate(_shots(case, seed)):
            m = [d[q].double().requires_grad_(True) for q in ("vp", "vs", "rho")]
            t, _ = _sim2(case, d, "VS", True, m)
            j = 0.5 * ((t - _observed(case, d, 1000 * seed + s).double()) ** 2).sum()
            grads.append([g.detach() for g in torch.autograd.grad(j, m)])
            total += float(j)
        return [total] + grads
    d = _inputs3(case, seed)
    if k == "spml3d":
        t, fields = _sim_spml(case, d)
        return [t] + fields
    if k == "grad3d":
        m = [d[q].double().requires_grad_(True) for q in ("vp", "vs", "rho")]
        t, _ = _sim3(case, d, m)
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        res = torch.randn(t.shape, generator=g, device=DEV)
        return [t.detach()] + list(torch.autograd.grad(t, m, res.double()))
    t, fields = _sim3(case, d, after=_layer(case, *_net(case, seed)) if k == "learned3d" else None)
    return [t] + fields
