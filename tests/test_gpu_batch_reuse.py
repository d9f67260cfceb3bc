"""A job whose last read set was empty takes the next one in a batch or a
server step like a new job."""
import pytest

import cases as G
import empanada_b200 as emp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("empty", [b"", G.fastq(["ACGTNACGTACG" * 4])])
@pytest.mark.parametrize("first", ["alone", "batch"])
@pytest.mark.parametrize("then", ["batch", "server"])
def test_after_an_empty_set(engine, empty, first, then):
    fq = G.BY_NAME["tiny"].fastq()
    want = emp.run_bytes(fq, engine=engine, min_ovlp=31)[0]
    jobs = [engine.job(min_ovlp=31) for _ in range(3)]
    for j in jobs[:2]:
        j.feed(empty)
    if first == "alone":
        for j in jobs[:2]:
            j.run()
    else:
        engine.run_batch(jobs[:2])
    for j in jobs[:2]:
        assert j.output() == b""
        j.reset()
    for j in jobs:
        j.feed(fq)
    if then == "batch":
        engine.run_batch(jobs)
    else:
        with emp.Server(engine) as srv:
            for j in jobs:
                srv.submit(j)
            while sum(srv.counts()):
                srv.step()
    for j in jobs:
        assert j.status() == 0 and j.output() == want and j.stats()["n_reads"] > 0
        j.close()
