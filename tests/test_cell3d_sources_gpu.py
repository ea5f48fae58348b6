"""Sources and receivers of the per-cell 3D kernels.  A point force near a
grid's last z block against the staged passes, at every order and shape
(Elastic3D_SSG_CPML adds 5 to the source's indices, so the case takes them off);
a source outside the cells that the passes update against the CPU oracle; and
more receivers than the split-PML stress kernel has threads."""
import numpy as np
import pytest
import torch

from cases import case3d, oracle3d, product3d, to_np

pytestmark = pytest.mark.gpu

F3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")
SHAPES = [((22, 24, 32), 4), ((23, 25, 36), 5), ((31, 33, 60), 8), ((40, 23, 68), 6)]


def _run(c, path, nt):
    w = product3d(c)
    w._build_plan().set_path(path)
    w.run(nt)
    w.check_status()
    out = {f: to_np(getattr(w, f)).copy() for f in F3}
    out.update({f"mem{a}": to_np(m).copy() for a, m in enumerate(w._mem) if m is not None})
    out["data"] = to_np(w.data).copy()
    return out


@pytest.mark.parametrize("N", [1, 2, 3, 4])
@pytest.mark.parametrize("shape,npml", SHAPES)
def test_point_force_in_the_last_block(cuda, N, shape, npml):
    kw = dict(dx=10.0, dy=7.3, dz=11.0) if N % 2 else {}
    c = case3d(shape=shape, N=N, scheme="CPML", nt=40, npml=npml, seed=N, **kw)
    c["isz"] = shape[2] - npml - 2 - 5
    a, b = _run(c, "two_pass", 40), _run(c, "staged", 40)
    assert a.keys() == b.keys() and np.abs(a["vx"]).max() > 0
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


@pytest.mark.parametrize("scheme", ["TENSOR", "CPML"])
@pytest.mark.parametrize("N", [1, 4])
@pytest.mark.parametrize("shape,npml", SHAPES[:2])
def test_source_outside_the_updated_cells(cuda, scheme, N, shape, npml):
    for cell in ((shape[0] // 2, shape[1] // 2, shape[2] - 1), (shape[0] - 1, 0, shape[2] // 2)):
        c = case3d(shape=shape, N=N, scheme=scheme, nt=40, npml=npml, seed=N)
        c["isx"], c["isy"], c["isz"] = (q - (5 if scheme == "CPML" else 0) for q in cell)
        w = product3d(c)
        assert w._build_plan().info()["path"] == "two_pass"
        o = oracle3d(c, wavelet=to_np(w._wavelet).astype(np.float32))
        w.run(40)
        o.run(0, 40)
        for f in F3:
            assert to_np(getattr(w, f)).tobytes() == getattr(o, f).tobytes(), (cell, f)


def test_more_receivers_than_threads(cuda):
    c = case3d(shape=(11, 11, 11), N=1, scheme="SPML", nt=20, npml=3)
    c["isx"], c["isy"], c["isz"], c["rsx"], c["rsy"], c["rsz"] = 5, 5, 5, 6, 5, 5
    one, many = product3d(c), product3d(c)
    n = 20000
    lin = np.full(n, int(many._rec_lin[0]), np.int64)
    many._receivers = lambda: (0, lin)
    many.data = torch.zeros((20, n), dtype=torch.float32, device="cuda")
    for w in (one, many):
        w._build_plan().set_path("two_pass")
        w.run(20)
    want = to_np(one.data).reshape(20)
    assert np.abs(want).max() > 0
    assert (to_np(many.data) == want[:, None]).all()
