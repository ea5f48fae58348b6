"""bench.py names the kernels that ran and counts their launches from the
plan's own report, on the CPU."""
import bench

STAGED, CELL = "k3s_velocity + k3s_stress", "k3_velocity + k3_stress"


def test_run_kernels():
    d3, d2 = {"shape": (200, 200, 200)}, {"shape": (400, 400)}
    spml = dict(d3, scheme="SPML")
    assert bench.run_kernels(d3, {"path": "staged"}, 1000) == (STAGED, 2001)
    assert bench.run_kernels(d3, {"path": "two_pass"}, 1000) == (CELL, 2001)
    assert bench.run_kernels(d3, {"path": "fused"}, 1000) == ("k3_fused", 1001)
    assert bench.run_kernels(spml, {"path": "two_pass"}, 1000) == ("ks_velocity + ks_stress", 2000)
    assert bench.run_kernels(spml, {"path": "staged"}, 1000) == (STAGED, 2000)
    assert bench.run_kernels(d2, {"path": "two_pass", "last_run_tiles": 143}, 2000) == ("k2r_run", 1)
    assert bench.run_kernels(d2, {"path": "two_pass", "last_run_tiles": 0}, 2000) == ("k2_velocity + k2_stress", 4000)
