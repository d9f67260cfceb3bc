"""Host-driven rounds (tables too large for M): their records stay on the
device until the output is copied, or go through host memory when the device
has no room for them; chunk counts around one digit of the chunk sort."""
import random

import pytest

import cases as G
import empanada_b200 as emp
from oracle import bind

pytestmark = pytest.mark.gpu


def _set(seed, n, L, genome, sub=0.0):
    rng = random.Random(seed)
    return G.fastq(G._reads(rng, G._genome(rng, genome), n, L, sub))


# M between a few entries and all of them; 256 and 257 chunks of the first table
@pytest.mark.parametrize("n,L,genome,o,M", [(1024, 40, 4000, 12, 8), (1028, 40, 4000, 12, 8), (3000, 60, 5000, 20, 700),
                                            (3000, 60, 5000, 20, 5999), (5000, 33, 30000, 5, 3000), (2, 30, 60, 10, 2)])
def test_matches_oracle(engine, n, L, genome, o, M):
    fq = _set(n + M, n, L, genome, 0.002)
    try:
        want, st = bind.run(fq, o, 16 * M)
    except bind.OracleError:  # no progress in the reference's partition loops: refused here too
        with pytest.raises(emp.EmpError):
            emp.run_bytes(fq, engine=engine, min_ovlp=o, reduce_mem=16 * M)
        return
    got, gst = emp.run_bytes(fq, engine=engine, min_ovlp=o, reduce_mem=16 * M)
    assert got == want
    for k in ("n_rounds", "n_edges", "n_records", "edges"):
        assert gst[k] == st[k], k


def test_any_device_budget():
    """From one that holds everything down to one that is refused: the same bytes."""
    fq = _set(5, 20000, 60, 20000, 0.002)
    want = bind.run(fq, 20, 16 * 15000)[0]
    budget, done = 64 << 20, 0
    while True:
        with emp.Engine(0, hbm_budget_bytes=budget) as engine:
            try:
                got, _ = emp.run_bytes(fq, engine=engine, min_ovlp=20, reduce_mem=16 * 15000)
            except emp.EmpError:
                break
        assert got == want
        done += 1
        budget -= budget // 50
    assert done
