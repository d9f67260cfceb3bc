"""A hand-over to the sweep kernel after host-driven rounds: the room for
edges is what the bucket kernel's launch left of it, whatever the host-driven
rounds found; sizes that no buffer has are refused."""
import pytest

import cases as G
import empanada_b200 as emp
from empanada_b200 import _native
from test_gpu_handover import _fastq

pytestmark = pytest.mark.gpu


def _trace(path):
    """Kernel of the last launch of rounds and its first round."""
    head, first = open(path).read().splitlines()[:2]
    return ("sweep", int(first.split(",")[3])) if head.startswith("step") else ("bucket", int(first.split(",")[0]))


def test_after_host_rounds(tmp_path, monkeypatch):
    trace = tmp_path / "trace.csv"
    monkeypatch.setenv("EMP_COOP_TRACE", str(trace))
    fq = _fastq(7, 4_600_000, 50, 8_200_000, 0.004)

    with emp.Engine(0) as engine:
        def run(reduce_mem, **tuned):
            with engine.tuned(**tuned), engine.job(min_ovlp=20, reduce_mem=reduce_mem) as job:
                job.feed(fq)
                job.run()
                return job.output(), job.stats()

        _, st = run("8g")
        mem = 32 * st["n_unique"]  # M / 2 = the first round's tables: two host-driven rounds
        want, wst = run(mem, round_driver=1)
        got, st = run(mem)
        kernel, r1 = _trace(trace)
        assert kernel == "sweep" and r1 >= 4  # two host-driven rounds, two or more of the bucket kernel, a hand-over
        assert 2 * st["sfx_live"][1] > 9 << 20
        assert got == want and st["edges"] == wst["edges"]
        host, bucket, sweep = sum(st["edges"][:2]), sum(st["edges"][2:r1]), sum(st["edges"][r1:])
        assert min(host, bucket, sweep) > 0
        launches = st["gpu_launches"]
        for cap in (bucket // 2, bucket + sweep - 1, bucket + sweep, host + bucket, host + bucket + sweep):
            got, st = run(mem, edge_cap=cap)
            assert got == want, cap
            # it runs again only where the two launches' edges do not fit
            assert (st["gpu_launches"] > launches) == (cap < bucket + sweep), cap


@pytest.mark.parametrize("cap", [(1 << 40) + 1, 1 << 61, 1 << 62, (1 << 64) - 1])
def test_edge_buffers_that_no_device_holds(engine, cap):
    fq = G.BY_NAME["tiny"].fastq()
    for tuned in ({}, {"round_driver": 2}):
        with engine.tuned(edge_cap=cap, **tuned), pytest.raises(emp.EmpError) as e:
            emp.run_bytes(fq, engine=engine, min_ovlp=31)
        assert e.value.code == _native.EMP_E_NOMEM
    with engine.tuned(edge_cap=cap, round_driver=1):  # host-driven rounds take what they need
        got, _ = emp.run_bytes(fq, engine=engine, min_ovlp=31)
    assert got == emp.run_bytes(fq, engine=engine, min_ovlp=31)[0]
