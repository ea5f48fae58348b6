"""3D runs on large grids whose rows are no multiple of 16 bytes: sw_run steps
pitched copies with the staged kernels, sw_step the caller's arrays with the
per-cell kernels.  Same bits for every row remainder, both orders, both
schemes and with and without slabs, for runs in pieces around the shortest
pitched run, a model changed between runs, and a run without its own graph
captured by the caller."""
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
    out["data"] = to_np(w.data).copy()
    return out


def _same(a, b):
    assert a.keys() == b.keys()
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


def _stepped(c, nt, it0=0, w=None):
    w = w or product3d(c)
    for i in range(it0, it0 + nt):
        w.update_SSG(i)
    return w


CASES = [dict(shape=(130, 111, 105)), dict(shape=(113, 131, 102), N=1), dict(shape=(125, 115, 107), npml=20),
         dict(shape=(130, 111, 105), surface=(True, False, False, True, True, False)),
         dict(shape=(130, 111, 105), surface=(False,) * 6)]


@pytest.mark.parametrize("scheme", ["TENSOR", "CPML"])
@pytest.mark.parametrize("kw", CASES)
def test_pitched_run_equals_steps(cuda, scheme, kw):
    c = case3d(scheme=scheme, nt=40, **kw)
    w = product3d(c)
    w.run(40)
    assert w._plan.info()["path"] == "two_pass"
    _same(_state(w), _state(_stepped(c, 40)))


def test_pieces_and_new_model(cuda):
    c = case3d(shape=(130, 111, 105), nt=60)
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
    c = case3d(shape=(130, 111, 105), nt=30)
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
