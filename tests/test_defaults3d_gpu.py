"""The defaults of 3D plans: the planes per work unit of the staged passes on
flat grids, where all units are alike and a few large ones beat many small, and
chosen again when the numeric mode changes unless the caller has chosen them;
and the path, by how the tiles fit the grid, with the other path's bits."""
import numpy as np
import pytest

from cases import case3d, product3d

pytestmark = pytest.mark.gpu


def _plan(shape, N=2, scheme="TENSOR", **kw):
    w = product3d(case3d(shape=shape, N=N, scheme=scheme, nt=4, hetero=False), **kw)
    return w, w._build_plan()


@pytest.mark.parametrize("N", [1, 2])
def test_flat_grids_take_large_units(cuda, N):
    for shape in ((300, 300, 40), (250, 200, 72)):
        w, p = _plan(shape, N)
        assert p.info()["path"] == "staged"
        # 252 and 268 us per step with 2 planes, 220 and 253 with these (order 2)
        assert p.info()["staged_chunk"] >= 10, shape
    w, p = _plan((100, 100, 100), N)
    assert p.info()["staged_chunk"] == 2


def test_units_follow_the_numeric_mode(cuda):
    shape = (300, 300, 40)  # exact: two CTAs per SM, fast: three
    exact = _plan(shape)[1].info()["staged_chunk"]
    w, p = _plan(shape, exact=False)
    fast = p.info()["staged_chunk"]
    assert fast != exact  # 200 us per step with 7 planes, 211 with the exact kernels' 20
    p.set_exact(True)
    assert p.info()["staged_chunk"] == exact
    p.set_exact(False)
    assert p.info()["staged_chunk"] == fast
    p.set_path("staged", 12)
    p.set_exact(True)
    assert p.info()["staged_chunk"] == 12


@pytest.mark.parametrize("shape,N,scheme,path", [
    ((230, 230, 40), 3, "TENSOR", "staged"), ((230, 230, 40), 4, "CPML", "staged"),
    ((230, 230, 40), 1, "SPML", "staged"), ((230, 230, 36), 2, "SPML", "two_pass"),
    ((240, 240, 36), 2, "SPML", "staged"),
    ((230, 230, 40), 3, "SPML", "two_pass"), ((230, 230, 40), 4, "SPML", "two_pass"),
    ((128, 128, 128), 3, "TENSOR", "staged"), ((128, 128, 128), 4, "TENSOR", "two_pass"),
    ((128, 128, 128), 1, "SPML", "two_pass"), ((160, 160, 80), 3, "TENSOR", "two_pass"),
    ((160, 160, 80), 1, "SPML", "staged"), ((160, 160, 80), 2, "SPML", "two_pass"),
    ((100, 100, 40), 3, "TENSOR", "two_pass"), ((60, 60, 40), 1, "SPML", "two_pass"),
    ((60, 60, 64), 2, "TENSOR", "staged"),
])
def test_default_path(cuda, shape, N, scheme, path):
    w, p = _plan(shape, N, scheme)
    assert p.info()["path"] == path
    o, q = _plan(shape, N, scheme)
    q.set_path("two_pass" if path == "staged" else "staged")
    for v in (w, o):
        v.run(4)
    for f in ("vx", "vz", "sxx", "syz"):
        a, b = getattr(w, f).cpu().numpy(), getattr(o, f).cpu().numpy()
        assert a.tobytes() == b.tobytes(), f
    assert np.abs(w.vx.cpu().numpy()).max() > 0
