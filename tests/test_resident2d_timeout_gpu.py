"""A tile of the 2D on-chip loop that gives up waiting for its rims (made to by
sw_plan_stop_on_chip: no wait really runs out) in a run's last step, where no
neighbour notices: the run's tiles agree, so every field and memory variable is
that from before the run, whichever tile it was; the status says so once,
run_checked raises, and the run repeats with the right bits."""
import numpy as np
import pytest
import torch

from cases import case2d, product2d, to_np
from seiswave_taichi_b200._native import SW_ERR_TIMEOUT, SeisWaveError

pytestmark = pytest.mark.gpu

F2 = ("vx", "vz", "sxx", "szz", "sxz")


def _state(w):
    out = {f: to_np(getattr(w, f)).copy() for f in F2}
    out.update({f"mem{a}": to_np(m).copy() for a, m in enumerate(w._mem) if m is not None})
    return out


def _same(a, b):
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_a_tile_that_gives_up(cuda, dtype):
    c = case2d(shape=(200, 190), dtype=dtype, nt=60, nrec=5, MT="explosive", src_scale=1e5)
    w, ref = product2d(c), product2d(c)
    ref.run(60)
    plan = w._plan(0)
    w.run(40)
    plan.status(w._stream())
    before, n = _state(w), plan.info()["on_chip_tiles"]
    assert n > 8
    for tile in (0, n // 2, n - 1):
        plan.stop_on_chip(tile)
        w.run(20, it0=40)
        with pytest.raises(SeisWaveError) as e:
            plan.status(w._stream())
        assert e.value.code == SW_ERR_TIMEOUT
        _same(before, _state(w))
        plan.status(w._stream())  # reported once
    plan.stop_on_chip(1)
    with pytest.raises(SeisWaveError):
        w.run_checked(20, it0=40, every=20)
    _same(before, _state(w))
    w.run_checked(20, it0=40, every=20)
    _same(_state(ref), _state(w))
    assert torch.equal(ref.data, w.data)


def test_stop_arguments(cuda):
    w = product2d(case2d(nt=20))
    plan = w._plan(0)
    for tile in (-1, plan.info()["on_chip_tiles"]):
        with pytest.raises(SeisWaveError):
            plan.stop_on_chip(tile)
