"""Solvers on streams of their own: a plan built and first run on a side stream
while another host thread keeps the default stream busy gives the bits of one
that has the device to itself (the device words of a plan are zero before any
stream can reach them); several 2D solvers whose on-chip loops share the device
keep their bits; a loop that the device refuses to hold is replayed; and a
plan's first run, which allocates its scratch, leaves another thread's stream
capture whole."""
import threading

import pytest
import torch

from cases import case2d, case3d, product2d, product3d, to_np

pytestmark = pytest.mark.gpu

F2 = ("vx", "vz", "sxx", "szz", "sxz")
F3 = ("vx", "vy", "vz", "sxx", "syy", "szz", "sxy", "sxz", "syz")


class _Busy:
    """Another host thread that always has work queued on the default stream."""

    def __enter__(self):
        self.stop = threading.Event()
        self.started = threading.Event()
        self.thread = threading.Thread(target=self._work)
        self.thread.start()
        assert self.started.wait(60)

    def _work(self):
        a = torch.randn(4096, 4096, device="cuda")
        queued = []
        while not self.stop.is_set():
            a = (a @ a).clamp_(-1, 1)
            queued.append(torch.cuda.Event())
            queued[-1].record()
            self.started.set()
            if len(queued) > 4:
                queued.pop(0).synchronize()
        torch.cuda.current_stream().synchronize()

    def __exit__(self, *_):
        self.stop.set()
        self.thread.join()


def _state(w, plan, fields):
    plan.status(w._stream())
    out = {f: to_np(getattr(w, f)).copy() for f in fields}
    out["data"] = to_np(w.data).copy()
    return out


def _run3(c, path, **kw):
    w = product3d(c, **kw)
    plan = w._build_plan()
    if path:
        plan.set_path(path)
    w.run(c["nt"])
    return _state(w, plan, F3)


def _run2(c, path, graph=True):
    w = product2d(c)
    plan = w._plan(0)
    plan.set_path(path)
    w.run(c["nt"], use_graph=graph)
    return _state(w, plan, F2)


@pytest.mark.parametrize("run,case", [
    (lambda c: _run3(c, "staged"), lambda: case3d(shape=(40, 36, 44), nt=40)),
    (lambda c: _run3(c, "staged"), lambda: case3d(shape=(40, 36, 44), nt=40, scheme="SPML")),
    (lambda c: _run3(c, "fused"), lambda: case3d(shape=(40, 36, 44), nt=41)),
    (lambda c: _run3(c, None), lambda: case3d(shape=(130, 111, 105), nt=20)),
    (lambda c: _run2(c, "two_pass"), lambda: case2d(nt=60, nrec=5)),
    (lambda c: _run2(c, "persistent"), lambda: case2d(nt=60, nrec=5)),
], ids=["staged", "staged_spml", "fused", "pitched", "on_chip", "persistent"])
def test_first_run_on_a_side_stream(cuda, run, case):
    c = case()
    ref = run(c)
    torch.cuda.synchronize()
    with _Busy():
        for _ in range(6):
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                got = run(c)
            for k in ref:
                assert got[k].tobytes() == ref[k].tobytes(), k


def _solvers(n, blocks, shape=(121, 90), nt=120):
    out = []
    for k in range(n):
        w = product2d(case2d(shape=shape, nt=nt, nrec=5, seed=k, MT="explosive", src_scale=1e5))
        w.set_on_chip(blocks)
        out.append(w)
    return out


@pytest.mark.parametrize("blocks", [-1, 20, 1])
def test_several_solvers_on_streams(cuda, blocks):
    refs = _solvers(6, 0)
    for w in refs:
        w.run(w.nt)
        assert w._plans[0].info()["on_chip_tiles"] == 0
    ws = _solvers(6, blocks)
    streams = [torch.cuda.Stream() for _ in ws]
    torch.cuda.synchronize()
    for w, s in zip(ws, streams):
        with torch.cuda.stream(s):
            w.run(50)
            w.run(w.nt - 50, it0=50)
    torch.cuda.synchronize()
    for w, r in zip(ws, refs):
        tiles = w._plans[0].info()["on_chip_tiles"]
        assert 0 < tiles <= (blocks if blocks > 0 else 1000) or blocks == 1
        a, b = _state(w, w._plans[0], F2), _state(r, r._plans[0], F2)
        for k in a:
            assert a[k].tobytes() == b[k].tobytes(), k


def test_refused_launch_is_replayed(cuda):
    """More tiles than the device has SMs can never be resident at once: the
    cooperative launch is refused, and the run replays the two launches."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    (ref,), (w,) = _solvers(1, 0, shape=(403, 391)), _solvers(1, 4 * sms, shape=(403, 391))
    ref.run(ref.nt)
    assert w._plan(0).info()["on_chip_tiles"] > sms
    w.run(60)
    assert w._plan(0).info()["on_chip_tiles"] == 0
    w.run(w.nt - 60, it0=60)
    a, b = _state(w, w._plan(0), F2), _state(ref, ref._plan(0), F2)
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


def test_small_grids_leave_room(cuda):
    """A small grid takes no more SMs than save it time, so that several
    solvers' on-chip loops can be resident at once."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for shape, n in (((60, 64), 8), ((121, 90), 4), ((160, 160), 2)):
        (w,) = _solvers(1, -1, shape=shape)
        assert 0 < n * w._plan(0).info()["on_chip_tiles"] <= sms


@pytest.mark.parametrize("case", [
    lambda: (product2d(case2d(nt=60, nrec=5)), "vz", lambda w: w.run(60)),
    lambda: (product3d(case3d(shape=(130, 111, 105), nt=20)), "vz", lambda w: w.run(20, use_graph=False)),
], ids=["on_chip", "pitched"])
def test_first_run_beside_a_capture(cuda, case):
    (ref, f, run), (w, _, _) = case(), case()
    run(ref)
    plan = w._plan(0) if hasattr(w, "_plans") else w._build_plan()  # built before the capture
    s = torch.cuda.Stream()
    x = torch.ones(1000, device="cuda")
    torch.cuda.synchronize()
    failed = []

    def other():
        try:
            with torch.cuda.stream(s):
                run(w)
        except Exception as e:  # noqa: BLE001 - reported below
            failed.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):  # the global mode
        x += 1
        t = threading.Thread(target=other)
        t.start()
        t.join()
        x *= 2
    assert not failed
    g.replay()
    torch.cuda.synchronize()
    plan.status()
    assert x.unique().tolist() == [4.0]
    assert to_np(getattr(w, f)).tobytes() == to_np(getattr(ref, f)).tobytes()
    assert to_np(w.data).tobytes() == to_np(ref.data).tobytes()


@pytest.mark.parametrize("shape,fits", [((121, 90), 4), ((200, 200), 1), ((400, 400), 1), ((700, 400), 1)])
def test_runs_in_flight_share_the_device(cuda, shape, fits):
    """Runs that meet others in flight on other streams take their share of the
    SMs (or, too large for it, are replayed, or wait for the whole device), the
    first of the next burst too; alone again a solver takes its own tiles.  Same
    bits throughout."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, nt = 6, 60
    ref = _solvers(1, 0, shape, nt)[0]
    ref.run(nt)
    want = _state(ref, ref._plans[0], F2)
    ws = [product2d(case2d(shape=shape, nt=nt, nrec=5, seed=0, MT="explosive", src_scale=1e5)) for _ in range(n)]
    plans = [w._plan(0) for w in ws]
    own = plans[0].info()["on_chip_tiles"]

    def alone():
        for _ in range(8):  # one stream: each run behind the last, not beside it
            ws[-1].run(4)
        assert plans[-1].info()["last_run_tiles"] == own

    alone()
    streams = [torch.cuda.Stream() for _ in range(n)]
    for burst in range(2):
        torch.cuda.synchronize()
        for q, (w, s) in enumerate(zip(ws, streams)):
            with torch.cuda.stream(s):
                torch.cuda._sleep(2_000_000_000)  # a second: its run is in flight for the others
                w.reset()
                w.run(nt)
            last = plans[q].info()["last_run_tiles"]
            met = q + 1 if burst == 0 else n
            if met <= fits or shape == (700, 400):  # that grid runs in turn, on the whole device
                assert last == own
            else:
                assert last <= sms // met
                assert last > 0 or shape == (400, 400)
        for w, p, s in zip(ws, plans, streams):
            with torch.cuda.stream(s):
                got = _state(w, p, F2)
            for k in want:
                assert got[k].tobytes() == want[k].tobytes(), k
    alone()
    torch.cuda.synchronize()
