"""The passes over the pairs that the run's statistics count are those that its sorts make."""
import pytest

import empanada_b200 as emp
from test_gpu_sweep import _set

pytestmark = pytest.mark.gpu


# one group in shared memory; a digit pass and groups; two digit passes and groups
# (more than 8 bits of groups from 2 * reads >> 8 = 2901 on)
@pytest.mark.parametrize("reads,passes", [(500, 1), (2048, 1), (2049, 2), (20_000, 2), (371_327, 2), (371_328, 3)])
def test_passes(engine, reads, passes):
    with engine.tuned(dedup_driver=1):
        _, st = emp.run_bytes(_set(reads, reads, 40, 10 * reads), engine=engine, min_ovlp=31)
    assert st["n_reads"] == reads
    assert (st["sort_passes"], st["sort_pass_elems"]) == (passes, passes * 2 * reads)
    assert st["ms_sort_passes"] > 0
