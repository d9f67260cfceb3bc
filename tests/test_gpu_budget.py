"""Batches and server steps under a device-memory budget, from one that holds
everything down to one that holds nothing: every job comes back with a status
of its own, and what ran has the bytes it gives alone."""
import random

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


@pytest.mark.parametrize("server", [True, False])
def test_a_job_that_does_not_fit_fails_alone(server):
    """Two small sets and then a large one: from the largest budget that
    refuses the large one's rounds, the small ones run."""
    rng = random.Random(3)
    small, large = (G.fastq(G._reads(rng, G._genome(rng, 10 * n), n, 100)) for n in (200, 8000))
    with emp.Engine(0) as engine:
        want = [emp.run_bytes(d, engine=engine, min_ovlp=31)[0] for d in (small, large)]
    budget = (8 << 20) + 16 * len(large)
    while True:
        with emp.Engine(0, hbm_budget_bytes=budget) as engine, engine.tuned(edge_cap=1 << 16):
            jobs = [engine.job(min_ovlp=31) for _ in range(3)]
            for j, d in zip(jobs, (small, small, large)):
                j.feed(d)
            (_serve if server else _batch)(engine, jobs)
            status = [j.status() for j in jobs]
            out = [j.output() if j.status() == 0 else None for j in jobs]
            for j in jobs:
                j.close()
        assert status[:2] == [0, 0], budget
        assert out[:2] == [want[0]] * 2
        if status[2]:
            break
        assert out[2] == want[1]
        budget -= budget // 200
    assert status[2] == _native.EMP_E_NOMEM


def test_a_batch_needs_little_more_than_its_jobs():
    """The least budget of two jobs as a batch, beside that of the two run one
    after another: what the batch shares beyond their own buffers is a few
    hundred bytes a job and 8 bytes a block of its launches."""
    rng = random.Random(4)
    sets = [G.fastq(G._reads(rng, G._genome(rng, 10 * n), n, 100)) for n in (700, 900)]

    def runs(budget, batch):
        try:
            with emp.Engine(0, hbm_budget_bytes=budget) as engine, engine.tuned(edge_cap=1 << 13):
                jobs = [engine.job(min_ovlp=31) for _ in sets]
                for j, d in zip(jobs, sets):
                    j.feed(d)
                if batch:
                    engine.run_batch(jobs)
                else:
                    for j in jobs:
                        j.run()
                return True
        except emp.EmpError as e:
            assert e.code == _native.EMP_E_NOMEM
            return False

    def least(batch):
        lo, hi = 1 << 16, 32 << 20  # refused, enough
        assert runs(hi, batch) and not runs(lo, batch)
        while hi - lo > 4096:
            mid = (lo + hi) // 2
            lo, hi = (lo, mid) if runs(mid, batch) else (mid, hi)
        return hi

    assert least(True) <= least(False) + (256 << 10)
