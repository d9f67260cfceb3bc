"""Batches and server steps under a device-memory budget, from one that holds
everything down to one that holds nothing: every job comes back with a status
of its own, and what ran has the bytes it gives alone."""
import pytest

import cases as G
import empanada_b200 as emp
from empanada_b200 import _native

pytestmark = pytest.mark.gpu

NAMES = ("tiny", "odd_len", "dups_palindromes")


def _outputs():
    with emp.Engine(0) as engine:
        return [emp.run_bytes(G.BY_NAME[n].fastq(), engine=engine, min_ovlp=31)[0] for n in NAMES]


def _burst(budget, run):
    """The sets fed to an engine of that budget and run: statuses and outputs (None: they cannot be fed)."""
    with emp.Engine(0, hbm_budget_bytes=budget) as engine, engine.tuned(edge_cap=1 << 13):
        jobs = []
        try:
            for n in NAMES:
                jobs.append(engine.job(min_ovlp=31))
                jobs[-1].feed(G.BY_NAME[n].fastq())
        except emp.EmpError:
            return None
        else:
            if not run(engine, jobs):
                return None
            return [(j.status(), j.output() if j.status() == 0 else None) for j in jobs]
        finally:
            for j in jobs:
                j.close()


def _serve(engine, jobs):
    back = []
    try:
        srv = emp.Server(engine, hbm_budget_bytes=1 << 40)
    except emp.EmpError:  # no room for its launch descriptors
        return False
    with srv:
        for j in jobs:
            srv.submit(j)
        for _ in range(20):
            back += srv.step()
            if not sum(srv.counts()):
                break
        assert not sum(srv.counts())
    assert sorted(j.handle.value for j in back) == sorted(j.handle.value for j in jobs)
    return True


def _batch(engine, jobs):
    try:
        engine.run_batch(jobs)
    except emp.EmpError as e:
        assert e.code == _native.EMP_E_NOMEM
    return True


@pytest.mark.parametrize("run", [_serve, _batch])
def test_every_job_comes_back(run):
    want = _outputs()
    budget, seen = 24 << 20, set()
    while (got := _burst(budget, run)) is not None:
        for (status, out), w in zip(got, want):
            assert status in (0, _native.EMP_E_NOMEM)
            assert status or out == w
        seen.add(sum(status == 0 for status, _ in got))
        budget -= budget // 30
    assert {0, len(NAMES)} <= seen
