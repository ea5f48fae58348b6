"""The split-field PML on the staged tiles against the one-thread-per-cell
kernels, which share no code with it above the quotient helpers: every field,
split part and trace, bit for bit.  Slab widths of both parities (pairs of
split parts lie at even and odd positions of the shell, across its parts'
borders and half outside it), both tile widths, open sides, every order, and a
damping profile whose divisors leave the corrected quotient's range."""
import numpy as np
import pytest

from cases import case3d, product3d, to_np

pytestmark = pytest.mark.gpu

F3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")

CASES = [
    dict(shape=(40, 36, 44), npml=8), dict(shape=(39, 35, 44), npml=7), dict(shape=(31, 33, 36), npml=5, N=1),
    dict(shape=(41, 30, 80), npml=9, N=3), dict(shape=(37, 34, 40), npml=6, N=4),
    dict(shape=(40, 36, 44), npml=7, surface=(True, False, True, False, False, True)),
    dict(shape=(40, 36, 44), npml=8, surface=(True, True, True, True, False, False)),
]


def _run(c, path, nt):
    w = product3d(c)
    plan = w._build_plan()
    plan.set_path(path)
    w.run(nt)
    plan.status(w._stream())
    out = {f: to_np(getattr(w, f)) for f in F3}
    out["split"], out["data"] = to_np(w._split), to_np(w.data)
    return out


@pytest.mark.parametrize("kw", CASES)
def test_staged_split_pml_equals_per_cell_kernels(cuda, kw):
    c = case3d(scheme="SPML", nt=80, **kw)
    a, b = _run(c, "staged", 80), _run(c, "two_pass", 80)
    assert np.abs(a["split"]).max() > 0
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


def test_divisors_outside_the_corrected_range(cuda):
    c = case3d(scheme="SPML", nt=40, npml=8)
    c["pml"]["vp_max"] = 1e13  # 1 + dt/2 d above 2^20 in the outer cells
    a, b = _run(c, "staged", 3), _run(c, "two_pass", 3)
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k
