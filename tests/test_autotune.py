"""The near-field tuner on a stand-in for the device: it times each setting that the kernels tell apart
once (a tile's limit is an eighth of the setting, 32 to 128 records; the threads per target have no
effect), and keeps the fastest.  No GPU."""
import pytest

from bit_b200 import autotune


class Device:
    """A context and its tree: the near field takes `seconds[records of a warp]`."""

    def __init__(self, seconds):
        self.seconds, self.config, self.timed = seconds, None, []

    def set_near_config(self, tile=0, threads_per_target=0):
        self.config = (tile, threads_per_target)

    def treemake(self, *a):
        return self

    def treemoments(self, *a):
        pass

    def evaluate(self, prm):
        self.timed.append(self.config)

    def stats(self):
        return {"t_near": self.seconds[min(128, max(32, self.config[0] // 8))]}

    def treeempty(self):
        pass


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("fastest", [32, 64, 128])
def test_tune_near_times_distinct_settings(precision, fastest):
    autotune._cache.clear()
    dev = Device({r: 1.0 if r == fastest else 2.0 for r in (32, 64, 128)})
    best, times = autotune.tune_near(dev, 5, 1, 1000, 0.5, 100, precision=precision, repeats=2)
    records = [min(128, max(32, tile // 8)) for tile, _ in times]
    assert sorted(records) == [32, 64, 128]
    assert all(split == 0 for _, split in times)
    assert len(dev.timed) == 2 * len(times)
    assert best == dev.config and best[0] // 8 == fastest
    assert autotune.tune_near(dev, 5, 1, 1000, 0.5, 100, precision=precision) == (best, times)
    autotune._cache.clear()
