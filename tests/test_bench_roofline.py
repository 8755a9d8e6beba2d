"""The benchmark's transport roofline counts one kind of launch: bytes, time and DRAM traffic per
application of the iterations that ran, whatever idle launches a batch ended with."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class FakeContext:
    def __init__(self, vox, its, idle, ms):
        self.bytes, self.count, self.ms = 78.0 * vox * its + 2.0 * vox, 2 * (its + idle), ms

    def timing_get(self, name):
        return self.ms, self.count

    def timing_bytes(self, name):
        return self.bytes


@pytest.mark.parametrize("idle", [0, 3, 40])
def test_figures_per_live_application(idle):
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    shape, its, ms = (10, 20, 30), [4, 3, 7], 1.5
    vox = 6000
    infos = [{"conc": {"iterations": n}, "acid": {"iterations": 0}} for n in its]
    r = bench.roofline(FakeContext(vox, sum(its), idle, ms), shape, infos)
    assert r["launches"] == 2 * sum(its) and r["launched"] == 2 * (sum(its) + idle)
    # 78 bytes a voxel and iteration, and 2 once
    assert r["bytes_per_launch"] == pytest.approx(39 * vox + vox / sum(its), abs=1)
    assert r["us_per_launch"] * r["launches"] == pytest.approx(1e3 * ms, rel=1e-2)
    assert r["traffic"] / r["bytes_per_launch"] == pytest.approx(39.71 / 39.0, rel=0.01)
    assert bench.roofline(FakeContext(vox, 0, 1, ms), shape, [infos[0] | {"conc": {"iterations": 0}}]) is None
