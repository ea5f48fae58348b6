"""The 2D loop that stays on the chip (sw_run of the SSG schemes, one
cooperative launch per run) against the two launches per step, which share no
code with it above the quotient helpers: every field, memory variable and
trace, bit for bit.  The cases sit at the edges of its tiling: the smallest
grids, one tile and many, widths around 32 and 64 columns, short and long
sides, slabs wider than a tile and no slabs, sources and receivers in corners
and rims, more receivers in a tile than its table holds, densities outside the
corrected quotient's range, the free-surface hook, runs in pieces, and a run
without its own graph captured by the caller."""
import numpy as np
import pytest
import torch

from cases import case2d, product2d, to_np

pytestmark = pytest.mark.gpu

F2 = ("vx", "vz", "sxx", "szz", "sxz")


def _state(w):
    out = {f: to_np(getattr(w, f)).copy() for f in F2}
    out.update({f"mem{a}": to_np(m).copy() for a, m in enumerate(w._mem) if m is not None})
    out["data"] = to_np(w.data).copy()
    return out


def _same(a, b):
    assert a.keys() == b.keys()
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


def _both(c, scheme, nt, pieces=None, **kw):
    got = []
    for graph in (True, False):
        w = product2d(c)
        it = 0
        for n in pieces or [nt]:
            w.run(n, it0=it, scheme=scheme, use_graph=graph, **kw)
            it += n
        for p in w._plans.values():
            p.status(w._stream())
        got.append(_state(w))
    _same(*got)
    return got[0]


CASES = [
    dict(shape=(11, 11), N=2, npml=3), dict(shape=(19, 23), N=4, npml=5), dict(shape=(16, 17), N=1, npml=4),
    dict(shape=(33, 32), N=2, npml=6), dict(shape=(97, 65), N=3, npml=20), dict(shape=(64, 129), N=2, npml=20),
    dict(shape=(301, 12), N=2, npml=4), dict(shape=(13, 640), N=1, npml=5), dict(shape=(260, 247), N=2, npml=20),
    dict(shape=(403, 391), N=2, npml=20), dict(shape=(150, 141), N=4, npml=12, dtype=np.float64),
    dict(shape=(61, 67), N=2, npml=10, dtype=np.float64), dict(shape=(90, 84), N=3, npml=10, surface=(True, False) * 2),
    dict(shape=(90, 84), N=2, npml=10, surface=(False,) * 4), dict(shape=(120, 75), N=2, dx=3.0, dz=7.3),
]


@pytest.mark.parametrize("scheme", ["VS", "SV"])
@pytest.mark.parametrize("kw", CASES)
def test_on_chip_loop_equals_two_launches(cuda, kw, scheme):
    nt = 60
    for mt in ("explosive", None):
        c = case2d(nt=nt, nrec=9, MT=mt, src_scale=1e5, **kw)
        _both(c, scheme, nt)


@pytest.mark.parametrize("cell", [(0, 0), (2, 2), (44, 44), (45, 46), (87, 3), (89, 83)])
def test_source_cell_anywhere(cuda, cell):
    for mt in ("explosive", None):
        c = case2d(shape=(90, 84), nt=40, nrec=5, MT=mt, src_scale=1e5)
        c["isx"], c["isz"] = cell
        s = _both(c, "VS", 40)
        assert np.abs(s["vz"]).max() > 0 or cell in ((0, 0), (89, 83))


def test_more_receivers_than_a_tile_holds(cuda):
    c = case2d(shape=(70, 60), nt=30, nrec=2, MT="explosive", src_scale=1e5)
    r = np.arange(1500)
    c["rsx"], c["rsz"] = (20 + r // 40 % 9).reshape(1, -1), (15 + r % 7).reshape(1, -1)
    _both(c, "VS", 30)


@pytest.mark.parametrize("rho", [1e-9, 3.1e7, 1e12])
def test_densities_outside_the_corrected_range(cuda, rho):
    c = case2d(shape=(80, 72), nt=50, nrec=5, MT="explosive", src_scale=1.0)
    c["rho"] = (c["rho"] / 2000.0 * rho).astype(np.float32)
    _both(c, "VS", 50)


def test_pieces_and_free_surface(cuda):
    c = case2d(shape=(100, 90), N=3, nt=60, nrec=5, MT="explosive", src_scale=1e5)
    whole = _both(c, "VS", 60)
    _same(whole, _both(c, "VS", 60, pieces=[7, 4, 1, 48]))
    c["isx"] = 3  # on the hooked layer
    _both(c, "VS", 60, free_surface=True)


def test_captured_run(cuda):
    c = case2d(shape=(100, 90), nt=30, nrec=5, MT="explosive", src_scale=1e5)
    ref = _both(c, "VS", 30)
    w = product2d(c)
    w.run(30)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        w.reset()
        w.run(30, use_graph=False)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    _same(ref, _state(w))
