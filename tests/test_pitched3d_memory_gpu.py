"""The pitched copies' memory: a run takes them only where they leave most of
the free memory to the caller, and not where the caller has chosen the per-cell
kernels; the bits are the same either way."""
import pytest
import torch

from cases import case3d, product3d, to_np

pytestmark = pytest.mark.gpu

F3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")
CASE = dict(shape=(130, 111, 105), nt=20)
COPIES = 12 * 130 * 111 * 108 * 4  # bytes, without the slabs


def _taken(w):
    """device bytes that the first run allocated"""
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    w.run(w.nt)
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


def _state(w):
    return {f: to_np(getattr(w, f)).tobytes() for f in F3}


def test_copies_only_with_room_to_spare(cuda):
    ref = product3d(case3d(**CASE))
    ref._build_plan()
    assert _taken(ref) >= COPIES
    w = product3d(case3d(**CASE))
    w._build_plan()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - 3 * COPIES, dtype=torch.uint8, device="cuda")
    assert _taken(w) < COPIES // 2
    del held
    torch.cuda.empty_cache()
    assert _state(w) == _state(ref)
    w.reset()
    assert _taken(w) >= COPIES  # room again


def test_no_copies_on_the_chosen_path(cuda):
    ref = product3d(case3d(**CASE))
    ref.run(20)
    w = product3d(case3d(**CASE))
    w._build_plan().set_path("two_pass")
    assert _taken(w) < COPIES // 2
    assert _state(w) == _state(ref)
    ref.reset()
    ref._plan.set_path("two_pass")  # after a pitched run
    ref.run(20)
    assert _state(w) == _state(ref)
