"""3D runs on grids whose rows are no multiple of 16 bytes: sw_run steps pitched
copies with the staged kernels, sw_step the caller's arrays with the two-pass
(split PML: per-cell) kernels.  Same bits for every row remainder, order,
scheme and slab set, for runs in pieces around the shortest pitched run, a
model changed between runs, and a captured run."""
import numpy as np
import pytest
import torch

from cases import case3d, product3d, to_np

pytestmark = pytest.mark.gpu

F3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")


def _state(w):
    w._plan.status(w._stream())
    out = {f: to_np(getattr(w, f)).copy() for f in F3}
    out.update({f"mem{a}": to_np(m).copy() for a, m in enumerate(w._mem) if m is not None})
    if w._split is not None:
        out["split"] = to_np(w._split).copy()
    out["data"] = to_np(w.data).copy()
    return out


def _same(a, b):
    assert a.keys() == b.keys()
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


def _stepped(c, nt, it0=0, w=None):
    w = w or product3d(c)
    step = w.update_SSG_SPML if c["scheme"] == "SPML" else w.update_SSG
    for i in range(it0, it0 + nt):
        step(i)
    return w


CASES = [dict(shape=(36, 30, 41)), dict(shape=(29, 33, 42), N=1), dict(shape=(34, 27, 39), N=3),
         dict(shape=(31, 32, 81), N=4, npml=6), dict(shape=(33, 30, 35), surface=(True, False, False, True, True, False)),
         dict(shape=(33, 30, 37), surface=(False,) * 6)]


@pytest.mark.parametrize("scheme", ["TENSOR", "CPML", "SPML"])
@pytest.mark.parametrize("kw", CASES)
def test_pitched_run_equals_steps(cuda, scheme, kw):
    c = case3d(scheme=scheme, nt=60, **kw)
    w = product3d(c)
    w.run(60)
    assert w._plan.info()["path"] == "two_pass"
    _same(_state(w), _state(_stepped(c, 60)))


def test_pieces_and_new_model(cuda):
    c = case3d(shape=(36, 30, 41), nt=60)
    w = product3d(c)
    it = 0
    for n in (5, 6, 1, 20, 28):
        w.run(n, it0=it, use_graph=n != 20)
        it += n
    ref = _stepped(c, 60)
    _same(_state(w), _state(ref))
    for v in (w, ref):
        v.set_model(c["vp"] * np.float32(1.05), c["vs"] * np.float32(0.97), c["rho"] * np.float32(1.1))
        v.reset()
    w.run(40)
    _same(_state(w), _state(_stepped(c, 40, w=ref)))


def test_captured_run(cuda):
    c = case3d(shape=(36, 30, 41), nt=30)
    w = product3d(c)
    w.run(30)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        w.reset()
        w.run(30, use_graph=False)
    g.replay()
    torch.cuda.synchronize()
    _same(_state(w), _state(_stepped(c, 30)))
