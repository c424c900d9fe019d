"""The roofline that bench.py reports."""
from __future__ import annotations

import bench

PEAKS = {"hbm_gbs": 6000.0, "bf16_tflops": 1600.0, "source": "test"}


def test_stencil_reports_the_runs_own_time_and_the_visited_tiles_rate():
    ks = {"k_temp_am": (5.0, 10), "k_diffuse_fs": (30.0, 10), "k_list": (2.0, 10)}
    r = bench._roofline(ks, 10, 1 << 24, "f32", PEAKS, (2.0, 0.25))
    assert r["kernel"] == "k_diffuse_fs"
    assert r["kernel_ms_per_launch"] == 3.0  # of the timed steps
    assert r["visited_fraction"] == 0.25
    assert abs(r["achieved"] - bench.BYTES_DIFFUSE_AM["f32"] * (1 << 24) * 0.25 / 2e-3 / 1e9) < 1e-6
    assert r["frac"] == r["achieved"] / 6000.0


def test_visits_are_those_of_single_steps():
    class Dom:
        calls = []
        maps = iter([(100, 50), (100, 70), (0, 0)])
        times = iter([3.0, 1.0, 2.0])

        def set_profiling(self, on):
            self.calls.append(on)

        def step(self, n):
            self.calls.append(n)

        def kernel_stats(self):
            return {"k_diffuse_fs": (next(self.times), 1)}

        def test_tile_map(self):
            return next(self.maps)

    ms, share = bench._stencil_visits(Dom(), 3)
    assert ms == 2.0 and abs(share - (0.5 + 0.3 + 1.0) / 3) < 1e-12
    assert Dom.calls == [True, 1, False] * 3
