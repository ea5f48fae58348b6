"""3D grids with more x planes than a launch grid's z extent (65535) on the
per-cell kernels: bit for bit the staged passes (float32) and the CPU oracle
(float64), with the source and a receiver among the last planes and every cell
in motion."""
import numpy as np
import pytest
import torch

from cases import case3d, oracle3d, product3d, to_np

pytestmark = pytest.mark.gpu

F3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")
NX = 65560


def _case(**kw):
    c = case3d(npml=2, nt=6, **kw)
    c["isx"] = NX - 12
    c["rsx"] = np.full_like(np.asarray(c["rsx"]), NX - 14) if np.ndim(c["rsx"]) else NX - 14
    return c


def _start(shape, dtype):
    rng = np.random.default_rng(3)
    return {f: (1e-3 * rng.standard_normal(shape)).astype(dtype) for f in F3}


def _run(c, path, start):
    w = product3d(c)
    w._build_plan().set_path(path)
    for f in F3:
        getattr(w, f).copy_(torch.from_numpy(start[f]))
    w.run(c["nt"])
    out = {f: to_np(getattr(w, f)) for f in F3}
    out["data"] = to_np(w.data)
    return out


@pytest.mark.parametrize("kw", [dict(scheme="SPML", N=1, shape=(NX, 12, 12)), dict(scheme="TENSOR", N=3, shape=(NX, 12, 12)),
                                dict(scheme="CPML", N=2, shape=(NX, 12, 12))])
def test_long_grid_equals_staged(cuda, kw):
    c = _case(**kw)
    start = _start(c["shape"], np.float32)
    a, b = _run(c, "two_pass", start), _run(c, "staged", start)
    assert np.abs(a["data"]).max() > 0
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


def test_long_grid_float64_equals_oracle(cuda):
    c = _case(N=1, shape=(NX, 9, 8), dtype=np.float64)
    start = _start(c["shape"], np.float64)
    w = product3d(c)
    w._build_plan()
    o = oracle3d(c, wavelet=to_np(w._wavelet).astype(np.float32))
    for f in F3:
        getattr(w, f).copy_(torch.from_numpy(start[f]))
        getattr(o, f)[...] = start[f]
    w.run(c["nt"])
    o.run(0, c["nt"])
    for f in F3:
        assert to_np(getattr(w, f)).tobytes() == getattr(o, f).tobytes(), f
