"""Which kernel runs a job's rounds, from the engine's trace of its launches:
the routes that other tests compare are the ones they name, and the shapes of
the bucket kernel choose no kernel."""
import hashlib

import pytest

import empanada_b200 as emp
import test_gpu_handover as handover
import test_gpu_parity as parity
import test_gpu_sweep as sweep
from cases import BY_NAME
from empanada_b200 import tune

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def traced(tmp_path_factory):
    """An engine that writes a trace, and the last launch's (kernel, [(first round, rounds) of a sweep step])."""
    path = tmp_path_factory.mktemp("trace") / "t.csv"
    with pytest.MonkeyPatch.context() as m:
        m.setenv("EMP_COOP_TRACE", str(path))
        engine = emp.Engine(0)

    def last():
        rows = [r.split(",") for r in path.read_text().splitlines()]
        if rows[0][0] != "step":
            return "bucket", int(rows[1][0])
        return "sweep", [(int(r[3]), int(r[4])) for r in rows[1:] if r[1] == "1"]

    yield engine, last
    engine.close()


@pytest.mark.parametrize("tuned", [{}, {"edge_cap": 8}, {"region_cap": 7}, {"region_cap": 40}, {"bucket_mean": 512}],
                         ids=str)
@pytest.mark.parametrize("name", ["tiny", "sub_errors", "dups_palindromes", "read_len_1"])
def test_the_bucket_kernel_for_every_round(traced, name, tuned):
    """region_cap: lists whose regions spill; bucket_mean: small buckets."""
    engine, last = traced
    with engine.tuned(round_driver=2, **tuned):
        _, out, _ = parity._run(engine, BY_NAME[name])
    assert hashlib.sha256(out).hexdigest() == parity.GOLDEN[name]["sha256"]
    assert last() == ("bucket", 0)


def test_the_bucket_kernel_with_more_buckets_than_shared_counters(traced):
    engine, last = traced
    with engine.tuned(round_driver=2, bucket_mean=512):
        _, out, _ = parity._run(engine, BY_NAME["larger"])
    assert hashlib.sha256(out).hexdigest() == parity.GOLDEN["larger"]["sha256"]
    assert last() == ("bucket", 0)


@pytest.mark.parametrize("tuned", [{"bucket_mean": 2175}, {"bucket_mean": 512}, {"region_cap": 40}], ids=str)
def test_bucket_shapes_choose_no_kernel(traced, tuned):
    engine, last = traced
    with engine.tuned(**tuned):
        _, out, _ = parity._run(engine, BY_NAME["sub_errors"])
    assert hashlib.sha256(out).hexdigest() == parity.GOLDEN["sub_errors"]["sha256"]
    assert last()[0] == "sweep"


@pytest.mark.parametrize("mean", [2900, 2175])
@pytest.mark.parametrize("name", sorted(handover.CASES))
def test_long_lists(traced, name, mean):
    engine, last = traced
    n, L, genome, sub, o, tuned = handover.CASES[name]
    with engine.job(min_ovlp=o, reduce_mem="8g") as job:
        job.feed(handover._fastq(n, n, L, genome, sub))
        with engine.tuned(bucket_mean=mean, **tuned):
            job.run()
        got, (kernel, at), job_unique = job.output(), last(), job.stats()["n_unique"]
        with engine.tuned(round_driver=2):
            job.run()
        assert job.output() == got
        assert last() == ("bucket", 0)
    assert tune.starts_in_sweep(job_unique, n) == (kernel == "sweep" and at[0][0] == 0)
    if name == "few_rounds":
        assert (kernel, at) == ("bucket", 0)
    else:
        assert kernel == "sweep" and (at[0][0] == 0) == (name == "sparse")  # handed over after some rounds, or not


@pytest.mark.parametrize("name", sorted(sweep.CASES))
def test_sweep_cases(traced, name):
    """Which of them retry a step, give the job to the bucket kernel, or start after host-driven rounds."""
    engine, last = traced
    make, o, reduce_mem = sweep.CASES[name]
    emp.run_bytes(make(), engine=engine, min_ovlp=o, reduce_mem=reduce_mem)
    kernel, steps = last()
    if name in ("crowded_group", "pairs_overflow"):
        assert (kernel, steps) == ("bucket", 0)
        return
    assert kernel == "sweep"
    assert (steps[0][0] > 0) == name.startswith("after_host_rounds")
    retried = any(a[0] == b[0] and a[1] > b[1] for a, b in zip(steps, steps[1:]))
    assert retried or name not in ("big_bin_retry", "low_complexity_20", "low_complexity_33")
