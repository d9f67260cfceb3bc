"""Unitigs by pointer jumping: path and cycle lengths at the powers of two
that decide the number of passes, both kinds together, against the oracle;
a graph that outlives its engine."""
import struct

import numpy as np
import pytest

import empanada_b200
from oracle import bind

pytestmark = pytest.mark.gpu


def _output(edges):
    """One record of shuffled edges."""
    f, t = edges[:, 0].astype(np.uint32), edges[:, 1].astype(np.uint32)
    return struct.pack("<Qi", len(edges), 40) + f.tobytes() + t.tobytes()


def _graph(paths, cycles, n_reads, seed):
    rng = np.random.default_rng(seed)
    ids = rng.permutation(2 * n_reads)
    edges, at = [], 0
    for length, closed in [(p, False) for p in paths] + [(c, True) for c in cycles]:
        x = ids[at:at + length]
        at += length
        edges.append(np.stack([x[:-1], x[1:]], 1))
        if closed:
            edges.append(np.array([[x[-1], x[0]]]))
    edges = np.concatenate(edges)
    return _output(edges[rng.permutation(len(edges))])


@pytest.mark.parametrize("paths,cycles,n_reads", [
    ([2], [], 1), ([1, 2, 3], [1], 4), ([4, 5, 7, 8, 9], [2, 3], 30), ([63, 64, 65], [31, 32, 33], 200),
    ([40_000], [], 20_000), ([], [40_000], 20_000), ([4095, 4096, 4097], [8191, 8192, 8193], 25_000),
    ([1000] * 50, [17] * 300, 40_000),
])
def test_lengths(engine, paths, cycles, n_reads):
    out = _graph(paths, cycles, n_reads, n_reads)
    order, starts = bind.unitigs(out, n_reads)
    with empanada_b200.Graph(engine, out, n_reads) as g:
        got, got_starts = g.unitigs()
        assert (got == order).all() and (got_starts == starts).all()
        st = g.stats()
    assert st["cycles"] == len(cycles) and st["unitigs"] == len(starts) - 1
    assert st["long_unitigs"] == int((np.diff(starts.astype(np.int64)) >= 2).sum())


def test_outlives_its_engine(tmp_path):
    out = _graph([100, 50], [9], 200, 3)
    order, starts = bind.unitigs(out, 200)
    eng = empanada_b200.Engine(0)
    g, unused = (empanada_b200.Graph(eng, out, 200) for _ in range(2))
    eng.close()
    got, got_starts = g.unitigs()
    assert (got == order).all() and (got_starts == starts).all()
    g.write_gfa(str(tmp_path / "g.gfa"), 60)
    assert (tmp_path / "g.gfa").read_bytes() == bind.gfa(out, 200, 60)
    g.close()
    unused.close()
