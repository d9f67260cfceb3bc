"""The sweep kernel (many rounds per step) against the oracle, byte for byte,
at the sizes where it can go wrong: a handful of reads, odd lengths, overlaps
down to zero bases, words that straddle, crowded groups that make a step
retry or hand the job to the bucket kernel, output bins too large for a warp,
and launches that follow host-driven rounds."""
import random

import pytest

import cases as G
import empanada_b200 as emp
from oracle import bind

pytestmark = pytest.mark.gpu


def _set(seed, n, L, genome, sub=0.0):
    rng = random.Random(seed)
    return G.fastq(G._reads(rng, G._genome(rng, genome), n, L, sub))


def _shared(seed, n_x, n_y, L=100, core=40):
    """n_x reads that end with one core, n_y that begin with it."""
    rng = random.Random(seed)
    c = G._genome(rng, core)
    return G.fastq([G._genome(rng, L - core) + c for _ in range(n_x)] + [c + G._genome(rng, L - core) for _ in range(n_y)])


def _low_complexity(seed, n, L):
    """Short repeats: equal keys within a read and between many reads, palindromes."""
    rng = random.Random(seed)
    return G.fastq(["".join(rng.choice(("A", "AC", "ACGT", "T", "GATC")) for _ in range(L))[:L] for _ in range(n)])


CASES = {
    "two_reads": (lambda: _set(1, 2, 40, 45), 10, 1 << 30),
    "one_warp": (lambda: _set(2, 33, 31, 200), 5, 1 << 30),
    "overlap_zero": (lambda: _set(3, 150, 17, 120), 0, 1 << 30),
    "all_rounds_one_word": (lambda: _set(4, 500, 16, 300), 2, 1 << 30),
    "one_round": (lambda: _set(5, 800, 64, 900), 63, 1 << 30),
    "longest_reads": (lambda: _set(6, 400, 512, 6000, 0.002), 21, 1 << 30),
    "odd_length_errors": (lambda: _set(7, 3001, 99, 4000, 0.01), 20, 1 << 30),
    "dense": (lambda: _set(8, 6000, 60, 1500), 20, 1 << 30),
    "low_complexity_20": (lambda: _low_complexity(9, 300, 20), 3, 1 << 30),
    "low_complexity_33": (lambda: _low_complexity(10, 700, 33), 1, 1 << 30),
    "big_bin_retry": (lambda: _shared(11, 1, 300), 31, 1 << 30),
    "pairs_overflow": (lambda: _shared(12, 150, 150), 31, 1 << 30),
    "crowded_group": (lambda: _shared(13, 2, 4500), 31, 1 << 30),
    "after_host_rounds": (lambda: _set(14, 5000, 80, 9000, 0.002), 25, 16 * 12000),
    "after_host_rounds_chunked": (lambda: _set(15, 4000, 75, 5000), 30, 16 * 3000),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_matches_oracle(engine, name):
    make, o, reduce_mem = CASES[name]
    fq = make()
    want, st = bind.run(fq, o, reduce_mem)
    got, gst = emp.run_bytes(fq, engine=engine, min_ovlp=o, reduce_mem=reduce_mem)
    assert got == want
    for k in ("n_reads", "n_rounds", "n_edges", "n_records", "sfx_live", "pfx_live", "edges"):
        assert gst[k] == st[k], k


def test_batch_of_all_with_the_bucket_kernel(engine):
    """Every case with in-core tables in one batch: as alone, and as the bucket kernel gives it."""
    sets = [(make(), o) for make, o, r in (CASES[k] for k in sorted(CASES)) if r == 1 << 30]
    want = [bind.run(fq, o)[0] for fq, o in sets]
    for tuned in ({}, {"bucket_mean": 2000}):
        with engine.tuned(**tuned):
            jobs = [engine.job(min_ovlp=o) for _, o in sets]
            for j, (fq, _) in zip(jobs, sets):
                j.feed(fq)
            engine.run_batch(jobs)
            got = [j.output() for j in jobs]
            for j in jobs:
                j.close()
        assert got == want
