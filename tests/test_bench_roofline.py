"""The roofline that bench.py reports."""
from __future__ import annotations

import bench

PEAKS = {"hbm_gbs": 6000.0, "bf16_tflops": 1600.0, "source": "test"}


def test_stencil_reports_the_runs_own_time_and_the_full_visits_rate():
    ks = {"k_temp_am": (5.0, 10), "k_diffuse_fs": (30.0, 10), "k_list": (2.0, 10)}
    r = bench._roofline(ks, 10, 1 << 24, "f32", PEAKS, 4.0)
    assert r["kernel"] == "k_diffuse_fs"
    assert r["kernel_ms_per_launch"] == 3.0  # tiles at rest left out
    assert r["all_tiles_ms_per_launch"] == 4.0
    assert abs(r["achieved"] - bench.BYTES_DIFFUSE_AM["f32"] * (1 << 24) / 4e-3 / 1e9) < 1e-6
    assert r["frac"] == r["achieved"] / 6000.0


def test_all_tiles_are_timed_in_steps_after_an_upload():
    class Dom:
        calls = []

        def download(self, f):
            return f

        def upload(self, f, v):
            self.calls.append("upload")

        def set_profiling(self, on):
            self.calls.append(on)

        def step(self, n):
            self.calls.append(n)

        def kernel_stats(self):
            return {"k_diffuse_fs": (0.25, 1)}

    assert bench._all_tiles_ms(Dom(), 3) == 0.25
    assert Dom.calls == ["upload", True, 1, False] * 3
