"""The autotuner's cache and candidates where the engine's choices changed
their meaning: entries of an earlier version, and which jobs are offered the
bucket kernel's tile size."""
import json

import pytest

from empanada_b200 import tune


class _Engine:
    def __init__(self):
        self.t = {"bucket_mean": 2900, "dedup_driver": 0}

    def tuning(self):
        return dict(self.t)

    def set_tuning(self, **c):
        self.t.update(c)


class _Job:
    def run(self):
        pass

    def output(self):
        return b"same"


@pytest.mark.parametrize("stamp", [{}, {"version": 1}, {"version": tune.VERSION + 1}, {"version": str(tune.VERSION)}])
def test_an_entry_of_another_version_is_timed_again(tmp_path, stamp):
    p = tmp_path / "tune.json"
    k = tune.shape_key("job", 1_200_000, 250)
    p.write_text(json.dumps({k: {"choice": {"bucket_mean": 1450}, "timings_ms": {"bucket_mean=1450": 1.0}, **stamp}}))
    eng = _Engine()
    r = tune.tune_job(eng, _Job(), 1_200_000, 250, cache=tune.Cache(str(p)), repeats=1)
    assert r["source"] == "timed" and eng.t["bucket_mean"] == 2900
    assert tune.Cache(str(p)).get(k) == r["choice"]


@pytest.mark.parametrize("reads,offered", [(1_000, False), (2_300_000, False), (2_400_000, True), (33_333_333, True)])
def test_tile_sizes_are_offered_to_long_lists(tmp_path, reads, offered):
    cache = tune.Cache(str(tmp_path / "t.json"))
    r = tune.tune_job(_Engine(), _Job(), reads, 150, cache=cache, repeats=1)
    assert any("bucket_mean" in label for label in r["timings_ms"]) == offered
    engine = _Engine()
    engine.run_batch = lambda jobs: None
    b = tune.tune_batch(engine, [_Job()] * 4, 4 * reads, 150, cache=cache)
    assert (b["source"] == "timed") == offered and (b["timings_ms"] is not None) == offered


def test_the_limits_are_the_engines():
    import os
    import re

    src = open(os.path.join(os.path.dirname(tune.__file__), "csrc", "kernels.h")).read()
    for name, value in (("kSweepMaxEntries", tune.SWEEP_MAX_ENTRIES), ("kSweepMaxSparse", tune.SWEEP_MAX_SPARSE)):
        a, b = re.search(name + r" = (\d+)ull << (\d+)", src).groups()
        assert int(a) << int(b) == value
    assert int(re.search(r"kSweepSparseR = (\d+)", src).group(1)) == tune.SWEEP_SPARSE_R
