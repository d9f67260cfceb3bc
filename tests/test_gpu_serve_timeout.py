"""A server step with a sweep launch and a bucket launch, one of which meets a
grid barrier that runs out of its wait (2 ms): the other's jobs are not touched."""
import pytest

import empanada_b200 as emp
from empanada_b200 import _native
from test_gpu_sweep import _set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [True, False])
def test_the_other_launch_goes_on(engine, first):
    small, large = _set(1, 300, 60, 3000), _set(2, 6000, 80, 60000)
    want = [emp.run_bytes(d, engine=engine, min_ovlp=31)[0] for d in (small, large)]
    jobs = [engine.job(min_ovlp=31) for _ in range(2)]
    for j, d in zip(jobs, (small, large)):
        j.feed(d)
    with emp.Server(engine, rounds_per_launch=5, rounds_per_launch_idle=5, share_min_entries=5000) as srv:
        for j in jobs:
            srv.submit(j)
        srv.step()
        assert srv.counts() == (0, 2, 0)
        if first:  # the sweep launch
            with engine.tuned(wait_limit_ns=2_000_000, block_next_wait=1), pytest.raises(_native.EmpError) as e:
                srv.step()
            assert e.value.code == _native.EMP_E_TIMEOUT
            assert jobs[0].status() == _native.EMP_E_TIMEOUT and srv.counts() == (0, 1, 0)
        else:  # the next bucket launch, with nothing else in flight
            assert srv.step() == [jobs[0]] and srv.counts() == (0, 1, 0)
            with engine.tuned(wait_limit_ns=2_000_000, block_next_wait=1), pytest.raises(_native.EmpError) as e:
                srv.step()
            assert e.value.code == _native.EMP_E_TIMEOUT
            assert jobs[1].status() == _native.EMP_E_TIMEOUT and srv.counts() == (0, 0, 0)
        while sum(srv.counts()):
            srv.step()
    bad = jobs[0] if first else jobs[1]
    for j, w in zip(jobs, want):
        if j is not bad:
            assert j.status() == 0 and j.output() == w
    bad.run()
    assert bad.output() == want[jobs.index(bad)]
    for j in jobs:
        j.close()
