"""Batches and server steps go on while a large copy to the device is in
flight: nothing that they put on their stream waits for the copy engine."""
import pytest
import torch

import cases as G
import empanada_b200 as emp
from test_gpu_sweep import _set

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def copy():
    """Starts a copy of about 70 ms and returns the event that ends it."""
    host = torch.empty(4 << 30, dtype=torch.uint8, pin_memory=True)
    dev = torch.empty_like(host, device="cuda")
    stream = torch.cuda.Stream()

    def start():
        torch.cuda.synchronize()
        end = torch.cuda.Event()
        with torch.cuda.stream(stream):
            dev.copy_(host, non_blocking=True)
            end.record()
        return end

    yield start
    torch.cuda.synchronize()


# every job in one sweep launch; a share of each job's rounds in bucket launches; both kinds in one step
@pytest.mark.parametrize("share_min", [None, 8_000_000, 1, 20_000])
def test_does_not_wait(engine, copy, share_min):
    sets = [_set(k, 400 * (k + 1), 80, 6000 * (k + 1), 0.002) for k in range(8)] + [G.BY_NAME["sub_errors"].fastq()] * 2
    jobs = [engine.job(min_ovlp=31) for _ in sets]
    want = [emp.run_bytes(d, engine=engine, min_ovlp=31)[0] for d in sets]
    for again in range(2):  # the first time without a copy: allocations and first launches
        for j, d in zip(jobs, sets):
            j.reset()
            j.feed(d)
        steps = [lambda: engine.run_batch(jobs)]
        if share_min is not None:
            srv = emp.Server(engine, rounds_per_launch=20, rounds_per_launch_idle=20, share_min_entries=share_min)
            for j in jobs:
                srv.submit(j)
            steps = [srv.step] * 6
        for step in steps:
            end = copy() if again else None
            step()
            assert end is None or not end.query()
        if share_min is not None:
            assert not sum(srv.counts())
            srv.close()
        assert [j.output() for j in jobs] == want
    for j in jobs:
        j.close()
