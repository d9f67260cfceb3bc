"""Pageable copies through the staging pieces, at sizes around the one from
which they are used and around whole pieces, both ways."""
import numpy as np
import pytest
import torch

import empanada_b200
from oracle import bind

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _reads(n, L, seed):
    """n reads of L bases as FASTQ bytes without names: 2 L + 5 bytes a record."""
    rng = np.random.default_rng(seed)
    rec = np.full((n, 2 * L + 5), ord("I"), np.uint8)
    rec[:, 0], rec[:, 1] = ord("@"), 10
    rec[:, 2:2 + L] = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, (n, L))]
    rec[:, 2 + L], rec[:, 3 + L], rec[:, 4 + L] = 10, ord("+"), 10
    rec[:, -1] = 10
    return rec.ravel()


@pytest.mark.parametrize("size", [4 * MIB - 1, 4 * MIB, 4 * MIB + 1, 5 * MIB + 12345, 23 * MIB + 7])
def test_feed_and_fingerprints(engine, size):
    L = 64
    fq = _reads(size // (2 * L + 5), L, size)
    fq = np.concatenate([fq[:1], np.full(size - fq.size, ord("n"), np.uint8), fq[1:]])  # a first name to fill up to the size
    want, n, _ = bind.fingerprints(fq)
    with engine.job(min_ovlp=60) as job:
        job.feed(fq)
        job.run()
        got = job.fingerprints()  # 16 bytes a read, pageable
    assert got.size == 2 * n and (got == want).all()


def test_output_pageable_as_page_locked(engine):
    rng = np.random.default_rng(3)
    genome = rng.integers(0, 4, 400_000)
    L = 50
    starts = rng.integers(0, genome.size - L, 900_000)
    fq = _reads(starts.size, L, 4).reshape(starts.size, -1)
    fq[:, 2:2 + L] = np.frombuffer(b"ACGT", np.uint8)[genome[starts[:, None] + np.arange(L)]]
    with engine.job(min_ovlp=20) as job:
        job.feed(fq.ravel())
        job.run()
        out = job.output()
        pinned = torch.zeros(len(out), dtype=torch.uint8, pin_memory=True).numpy()
        assert len(out) > 4 * MIB and job.output_into(pinned) == len(out)
    assert out == pinned.tobytes() == bind.run(fq.ravel(), 20)[0]


def test_graph_arrays(engine):
    n_reads = 1_300_000
    rng = np.random.default_rng(5)
    ids = rng.permutation(2 * n_reads).astype(np.uint32)
    f, t = ids[:-1:2], ids[1::2]
    out = np.uint64(f.size).tobytes() + np.int32(40).tobytes() + f.tobytes() + t.tobytes()
    order, starts = bind.unitigs(out, n_reads)
    with empanada_b200.Graph(engine, out, n_reads) as g:
        got, got_starts = g.unitigs()
    assert (got == order).all() and (got_starts == starts).all()
