"""The per-cell 3D kernels against the TMA-staged passes, which share no code
with them above the quotient helpers: every field, memory variable and trace,
bit for bit, for each order and scheme, at grids around the edges of their
blocks (32 z cells by 8 y cells), with and without slabs, and with a source on
a grid's last block."""
import numpy as np
import pytest

from cases import case3d, product3d, to_np
from seiswave_taichi_b200._native import SeisWaveError

pytestmark = pytest.mark.gpu

F3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")


def _run(c, path, nt):
    w = product3d(c)
    try:
        (w._plan or w._build_plan()).set_path(path)
    except SeisWaveError:
        pytest.skip(f"no {path} path with the source this close to the x edge")
    w.run(nt)
    w._plan.status(w._stream())
    out = {f: to_np(getattr(w, f)).copy() for f in F3}
    out.update({f"mem{a}": to_np(m).copy() for a, m in enumerate(w._mem) if m is not None})
    if getattr(w, "_split", None) is not None:
        out["split"] = to_np(w._split).copy()
    out["data"] = to_np(w.data).copy()
    return out


@pytest.mark.parametrize("scheme", ["TENSOR", "CPML", "SPML"])
@pytest.mark.parametrize("N", [1, 2, 3, 4])
@pytest.mark.parametrize("shape,npml", [((22, 24, 32), 4), ((23, 25, 36), 5), ((31, 33, 60), 8), ((40, 23, 68), 6)])
def test_per_cell_equals_staged(cuda, scheme, N, shape, npml):
    kw = dict(dx=10.0, dy=7.3, dz=11.0) if N % 2 else {}
    c = case3d(shape=shape, N=N, scheme=scheme, nt=40, npml=npml, seed=N, **kw)
    c["isz"] = shape[2] - npml - 2
    a, b = _run(c, "two_pass", 40), _run(c, "staged", 40)
    assert a.keys() == b.keys() and np.abs(a["vx"]).max() > 0
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k
