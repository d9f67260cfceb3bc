"""The sweep kernel's places for candidates and pairs, drawn from 1 to 16
counters by the job's size and share of the launch: below, at and above the
sizes where a counter is added, and jobs of unequal shares in one launch."""
import random

import pytest

import cases as G
import empanada_b200 as emp
from oracle import bind

pytestmark = pytest.mark.gpu


def _set(seed, n, L, genome):
    rng = random.Random(seed)
    return G.fastq(G._reads(rng, G._genome(rng, genome), n, L, 0.002))


@pytest.mark.parametrize("n", [4000, 8000, 8600, 17500, 34000, 68500])
def test_matches_oracle(engine, n):
    fq = _set(n, n, 44, 6 * n)
    want, st = bind.run(fq, 20)
    got, gst = emp.run_bytes(fq, engine=engine, min_ovlp=20)
    assert got == want and gst["edges"] == st["edges"]


def test_unequal_shares(engine):
    sets = [_set(k, n, 44, max(50, 5 * n)) for k, n in enumerate([60000, 30000, 9000, 200, 1])]
    jobs = [engine.job(min_ovlp=20) for _ in sets]
    for j, fq in zip(jobs, sets):
        j.feed(fq)
    engine.run_batch(jobs)
    got = [j.output() for j in jobs]
    for j in jobs:
        j.close()
    assert got == [bind.run(fq, 20)[0] for fq in sets]
