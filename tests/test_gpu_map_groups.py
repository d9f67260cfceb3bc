"""A batch whose FASTQ is still on its way goes through the map phase in
groups: the outputs are those of the jobs alone, a failing job among them
keeps its status, and so does one with other read lengths."""
import numpy as np
import pytest
import torch

import empanada_b200 as emp
from empanada_b200 import _native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [[0, 1, 2, 3, 4, 5, 6], [6, 3, 5, 0, 2, 1, 4], [1, 2, 3, 4, 5, 6, 0]])
@pytest.mark.parametrize("served", [False, True])
def test_groups(engine, order, served):
    reads = (700_000, 90_000, 20, 50_000, 150_000)  # 245 MB and less
    data = [synth.fastq_bytes(synth.Workload("set", seed=k, genome_len=max(400, 10 * n), n_reads=n, read_len=130 + k,
                                             sub_rate=0.001, min_ovlp=31)) for k, n in enumerate(reads)]
    data += [b"", b"@r\nACGTACGTAC\n+\nIIIIIIIIII\n@r\nACGTACG\n+\nIIIIIII\n"]  # nothing; two lengths
    want = []
    for d in data[:-1]:
        want.append(emp.run_bytes(d, engine=engine, min_ovlp=31)[0])
    jobs, held = {}, []
    for k in order:
        host = torch.empty(max(1, len(data[k])), dtype=torch.uint8, pin_memory=True).numpy()[:len(data[k])]
        host[:] = np.frombuffer(data[k], np.uint8)
        held.append(host)
        jobs[k] = engine.job(min_ovlp=31)
    for k, host in zip(order, held):
        jobs[k].feed_async(host)
    if served:
        with emp.Server(engine) as srv:
            for k in order:
                srv.submit(jobs[k])
            while sum(srv.counts()):
                srv.step()
    else:
        with pytest.raises(emp.EmpError) as e:
            engine.run_batch([jobs[k] for k in order])
        assert e.value.code == _native.EMP_E_FORMAT
    for k in order:
        if k == 6:
            assert jobs[k].status() == _native.EMP_E_FORMAT
        else:
            assert jobs[k].status() == 0 and jobs[k].output() == want[k]
        jobs[k].close()
