"""The 3D autotuner on plans without a staged path: nothing is timed or cached
for the per-cell kernels, which have no work units, and the units of runs on
pitched copies are tuned like the staged ones."""
import numpy as np
import pytest
import torch

from cases import case3d, product3d, to_np
from seiswave_taichi_b200.batch import cache_load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(scheme="SPML"), dict(N=4), dict(dtype=np.float64), dict(shape=(40, 36, 43))])
def test_per_cell_has_nothing_to_tune(cuda, tmp_path, monkeypatch, kw):
    cache = tmp_path / "autotune.json"
    monkeypatch.setenv("SEISWAVE_AUTOTUNE_CACHE", str(cache))
    w = product3d(case3d(nt=20, **kw))
    assert w._build_plan().info()["path"] == "two_pass"
    assert w.autotune() == 0 and not cache.exists()


def test_chosen_split_pml_tiles_are_tuned(cuda, tmp_path, monkeypatch):
    monkeypatch.setenv("SEISWAVE_AUTOTUNE_CACHE", str(tmp_path / "autotune.json"))
    c = case3d(nt=40, scheme="SPML")
    w, ref = product3d(c), product3d(c)
    w._build_plan().set_path("staged")
    w.run(20)
    split = w._split.clone()
    chunk = w.autotune(steps=3)
    assert chunk in w.AUTOTUNE_CHUNKS and w._plan.info()["staged_chunk"] == chunk
    assert torch.equal(w._split, split)
    w.run(20, it0=20)
    ref.run(40)
    assert to_np(w.vx).tobytes() == to_np(ref.vx).tobytes() and torch.equal(w._split, ref._split)


def test_pitched_runs_are_tuned(cuda, tmp_path, monkeypatch):
    monkeypatch.setenv("SEISWAVE_AUTOTUNE_CACHE", str(tmp_path / "autotune.json"))
    c = case3d(shape=(130, 111, 105), nt=40)
    w, ref = product3d(c), product3d(c)
    w.run(20)
    before = to_np(w.vz).tobytes()
    chunk = w.autotune(steps=3)
    assert chunk in w.AUTOTUNE_CHUNKS and w._plan.info()["staged_chunk"] == chunk
    assert to_np(w.vz).tobytes() == before and len(cache_load()) == 1
    w.run(20, it0=20)
    ref.run(40)
    assert to_np(w.vz).tobytes() == to_np(ref.vz).tobytes()
    again = product3d(c)
    assert again.autotune() == chunk and again._plan.info()["staged_chunk"] == chunk
    again._plan.set_path("two_pass")
    assert again.autotune() == 0
