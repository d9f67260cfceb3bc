"""Long lists: the bucket kernel's launch leaves its last rounds to the sweep
kernel, against all rounds in the bucket kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fastq(seed, n, L, genome, sub):
    rng = np.random.default_rng(seed)
    g = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, genome)]
    both = np.concatenate([g, np.frombuffer(bytes(range(256)).translate(bytes.maketrans(b"ACGT", b"TGCA")), np.uint8)[g][::-1]])
    rec = np.full((n, 2 * L + 5), ord("I"), np.uint8)
    rec[:, 0], rec[:, 1] = ord("@"), 10
    start = rng.integers(0, genome - L + 1, n) + genome * rng.integers(0, 2, n)
    rec[:, 2:2 + L] = both[start[:, None] + np.arange(L)]
    if sub:
        k = rng.integers(0, n * L, int(n * L * sub))
        rec[k // L, 2 + k % L] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, k.size)]
    rec[:, 2 + L], rec[:, 3 + L], rec[:, 4 + L] = 10, ord("+"), 10
    rec[:, -1] = 10
    return rec.ravel()


# sparse enough for the sweep kernel from the start; a long tail of errors;
# dense until few are left; too few rounds to hand over; an edge buffer that is
# too small
CASES = {
    "sparse": (2_600_000, 60, 60_000_000, 0.0, 30, {}),
    "errors": (3_400_000, 50, 6_000_000, 0.004, 20, {}),
    "dense": (3_300_000, 95, 6_000_000, 0.0, 20, {}),
    "few_rounds": (3_300_000, 34, 6_000_000, 0.0, 20, {}),
    "edge_buffer": (3_400_000, 50, 6_000_000, 0.004, 20, {"edge_cap": 4_500_000}),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_as_the_bucket_kernel_alone(engine, name):
    n, L, genome, sub, o, tuned = CASES[name]
    with engine.job(min_ovlp=o, reduce_mem="8g") as job:
        job.feed(_fastq(n, n, L, genome, sub))
        with engine.tuned(**tuned):
            job.run()
        got, st = job.output(), job.stats()
        with engine.tuned(bucket_mean=2800):
            job.run()
        want, wst = job.output(), job.stats()
    assert 2 * st["n_unique"] > 9 << 20
    assert got == want
    for k in ("n_rounds", "n_edges", "n_records", "sfx_live", "pfx_live", "edges"):
        assert st[k] == wst[k], k
