"""The work that users of this package have it do, as cases that can be timed.

Each case is one call sequence through the public entry points on seeded
synthetic reads: a uniform random genome (with repeat families where named),
reads at uniform positions, half of them reverse-complemented, uniform
substitutions, constant quality, written as FASTQ.  Read sets are made on the
GPU, so that preparing one costs less than running it.

A job case holds a fed job (FASTQ resident in HBM) and runs it, its output.bin
copied into page-locked host memory.  The other cases say what they run beside
them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import empanada_b200 as emp

_ENGINE = None


def _engine():
    """One engine per process and device, as a program keeps it."""
    global _ENGINE
    if _ENGINE is None:
        _ENGINE = emp.Engine(0)
    return _ENGINE


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest useful call: a plasmid-sized set, all latency and launches
        _job("job_tiny", reads=2_000, read_len=100, genome=40_000),
        # a bacterial sample at 15x with the default options
        _job("job_small", reads=100_000, read_len=150, genome=1_000_000),
        # 60x of 250 bp reads with sequencing errors, long minimum overlap: many rounds of long-lived entries
        _job("job_larger", reads=1_200_000, read_len=250, genome=5_000_000, sub=0.001, min_ovlp=75,
             reduce_mem="12g"),
        # odd length, errors, and reads that the N filter drops (real runs hold some)
        _job("job_n_reads", reads=400_009, read_len=251, genome=2_000_003, sub=0.001, n_frac=0.03),
        # the largest single job: 50x of a 100 Mbp genome with repeat families, HBM-sized blocks
        _job("job_repeats", reads=33_333_333, read_len=150, genome=100_000_000, repeats=0.05, reduce_mem="160g"),
        # the same at a tenth with -r 100m: tables larger than M, the chunked sort and split records
        _job("job_streamed", reads=3_333_333, read_len=150, genome=10_000_000, repeats=0.05, reduce_mem="100m"),
        # one call on FASTQ bytes in host memory, job made and dropped inside
        dict(name="one_shot_host", kind="host", reads=150_001, read_len=101, genome=1_000_000, sub=0.001, n_frac=0.0,
             repeats=0.0, min_ovlp=31, reduce_mem="1g"),
        # 256 independent read sets of 50-500 kbp genomes in one batch
        dict(name="batch_256", kind="batch", sets=256, genome_min=50_000, genome_max=500_000, len_min=100,
             len_max=300, cov_min=10.0, cov_max=80.0, sub=0.001, min_ovlp=31),
        # a burst of 48 requests from pinned host memory through the server
        dict(name="served_48", kind="served", sets=48, genome_min=50_000, genome_max=500_000, len_min=100,
             len_max=300, cov_min=10.0, cov_max=80.0, sub=0.001, min_ovlp=31),
        # the graph consumer: unitigs of a tenth of the largest job's overlaps
        dict(name="unitigs", kind="graph", reads=3_333_333, read_len=150, genome=10_000_000, sub=0.0, n_frac=0.0,
             repeats=0.05, min_ovlp=31, reduce_mem="4g"),
        # the fingerprint sort as an entry point of its own
        dict(name="sort_pairs", kind="sort", pairs=33_333_333),
        # the sort for callers that must not allocate
        dict(name="sort_static", kind="sort_static", pairs=1_000_003),
    ]


def _job(name, reads, read_len, genome, sub=0.0, n_frac=0.0, repeats=0.0, min_ovlp=31, reduce_mem="1g"):
    return dict(name=name, kind="job", reads=reads, read_len=read_len, genome=genome, sub=sub, n_frac=n_frac,
                repeats=repeats, min_ovlp=min_ovlp, reduce_mem=reduce_mem)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "job", "job", "job", "streamed", "host", "batch", "served", "graph", "sort",
                       "sort_static"])
    if kind == "sort":
        return dict(kind=kind, pairs=_log_int(rng, 1_000, 60_000_000))
    if kind == "sort_static":
        return dict(kind=kind, pairs=_log_int(rng, 500, emp.SORT_STATIC_MAX_PAIRS))
    if kind in ("batch", "served"):
        lo = _log_int(rng, 20_000, 100_000)
        return dict(kind=kind, sets=_log_int(rng, 4, 256 if kind == "batch" else 60), genome_min=lo,
                    genome_max=lo * rng.randint(2, 8), len_min=rng.randint(80, 140), len_max=rng.randint(150, 300),
                    cov_min=float(rng.randint(8, 20)), cov_max=float(rng.randint(30, 80)),
                    sub=rng.choice([0.0, 0.001, 0.002]), min_ovlp=rng.choice([25, 31, 45]))
    most = {"job": 12_000_000, "streamed": 3_000_000, "host": 1_000_000, "graph": 4_000_000}[kind]
    reads = _log_int(rng, 20_000 if kind in ("streamed", "graph") else 1_000, most)
    read_len = rng.randint(60, 300)
    genome = max(4 * read_len, int(reads * read_len / rng.uniform(10.0, 80.0)))
    min_ovlp = rng.choice([21, 31, 31, 45, read_len // 2])
    reduce_mem = rng.choice(["1g", "12g", "160g"])
    if kind == "streamed":  # M = reduce_mem / 16 between a sixth of the read-ends and all of them
        reduce_mem = str(int(32 * reads / rng.uniform(1.0, 6.0)))
    elif reads > 8_000_000 or kind == "graph":
        reduce_mem = "160g"
    return dict(kind="job" if kind == "streamed" else kind, reads=reads, read_len=read_len, genome=genome,
                sub=rng.choice([0.0, 0.0, 0.001, 0.003]), n_frac=rng.choice([0.0, 0.0, 0.02]) if kind != "graph" else 0.0,
                repeats=rng.choice([0.0, 0.05]) if genome >= 100_000 else 0.0, min_ovlp=min_ovlp,
                reduce_mem=reduce_mem)


# ---------------------------------------------------------------- synthetic reads
_COMPLEMENT = bytes.maketrans(b"ACGT", b"TGCA")


def _lut(table):
    return torch.tensor(list(table), dtype=torch.uint8, device="cuda")


def _genome(size, repeats, gen, host):
    """ACGT bytes; `repeats` of them covered by families of 1-5 kbp copies (2-50 each, 1% divergence)."""
    g = _lut(b"ACGT")[torch.randint(0, 4, (size,), generator=gen, device="cuda")]
    if repeats and size > 20_000:
        src, dst, fam_at, covered = [], [], 0, 0
        while covered < repeats * size:
            length = int(host.integers(1000, 5001))
            copies = min(int(host.integers(2, 51)), int((repeats * size - covered) // length) + 1)
            at = host.integers(0, size - length + 1, copies)
            dst.append((at[:, None] + np.arange(length)).ravel())
            src.append(np.tile(np.arange(fam_at, fam_at + length), copies))
            fam_at += length
            covered += copies * length
        fam = _lut(b"ACGT")[torch.randint(0, 4, (fam_at,), generator=gen, device="cuda")]
        src = fam[torch.from_numpy(np.concatenate(src)).cuda()]
        dst = np.concatenate(dst)
        # where copies overlap, the last one stays
        last = dst.size - 1 - np.unique(dst[::-1], return_index=True)[1]
        src, dst = src[torch.from_numpy(last).cuda()], torch.from_numpy(dst[last]).cuda()
        g[dst] = _substitute(src, 0.01, gen)
    return g


def _substitute(x, rate, gen):
    """Each byte replaced by another base with probability `rate` (in place)."""
    flat = x.view(-1)
    at = torch.nonzero(torch.rand(flat.shape, generator=gen, device="cuda") < rate).view(-1)
    code = torch.zeros(256, dtype=torch.long, device="cuda")
    for i, c in enumerate(b"ACGT"):
        code[c] = i
    shift = torch.randint(1, 4, at.shape, generator=gen, device="cuda")
    flat[at] = _lut(b"ACGT")[(code[flat[at].long()] + shift) & 3]
    return x


def _fastq(c, seed):
    """The read set's FASTQ as a uint8 tensor on the GPU."""
    n, L = int(c["reads"]), int(c["read_len"])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    G = max(int(c["genome"]), L)
    fwd = _genome(G, c["repeats"], gen, np.random.default_rng(seed))
    both = torch.cat([fwd, _lut(bytes(range(256)).translate(_COMPLEMENT))[fwd.long()].flip(0)])
    windows = both.as_strided((2 * G - L + 1, L), (1, 1))
    parts, lo, digits = [], 0, 1
    while lo < n:  # reads with names of the same length: records of one size
        hi = min(n, 10 ** digits)
        parts.append((lo, hi, digits))
        lo, digits = hi, digits + 1
    out = torch.empty(sum((hi - lo) * (7 + d + 2 * L) for lo, hi, d in parts), dtype=torch.uint8, device="cuda")
    at = 0
    for lo, hi, d in parts:
        rec = 7 + d + 2 * L  # "@r<i>\n" read "\n+\n" quality "\n"
        step = max(1, 48_000_000 // L)
        for i in range(lo, hi, step):
            m = min(step, hi - i)
            row = out[at:at + m * rec].view(m, rec)
            at += m * rec
            row[:, 0], row[:, 1] = ord("@"), ord("r")
            ids = torch.arange(i, i + m, device="cuda")
            for k in range(d):
                row[:, 2 + k] = (ids // 10 ** (d - 1 - k) % 10 + ord("0")).to(torch.uint8)
            start = torch.randint(0, G - L + 1, (m,), generator=gen, device="cuda")
            start += G * torch.randint(0, 2, (m,), generator=gen, device="cuda")  # either strand
            reads = windows[start]
            if c["sub"]:
                reads = _substitute(reads, c["sub"], gen)
            if c["n_frac"]:
                bad = torch.nonzero(torch.rand(m, generator=gen, device="cuda") < c["n_frac"]).view(-1)
                reads[bad, torch.randint(0, L, bad.shape, generator=gen, device="cuda")] = ord("N")
            s = 2 + d
            row[:, s] = 10
            row[:, s + 1:s + 1 + L] = reads
            row[:, s + 1 + L], row[:, s + 2 + L], row[:, s + 3 + L] = 10, ord("+"), 10
            row[:, s + 4 + L:s + 4 + 2 * L] = ord("I")
            row[:, s + 4 + 2 * L] = 10
    return out


def _sets(c, seed):
    """The read sets of a batch: genome log-uniform, read length and coverage uniform, fixed by the case's ranges."""
    rng = np.random.default_rng(4)
    out = []
    for k in range(c["sets"]):
        g = int(round(math.exp(rng.uniform(math.log(c["genome_min"]), math.log(c["genome_max"])))))
        L = int(rng.integers(c["len_min"], c["len_max"] + 1))
        n = max(1, int(g * rng.uniform(c["cov_min"], c["cov_max"]) / L))
        out.append(dict(reads=n, read_len=L, genome=g, sub=c["sub"], n_frac=0.0, repeats=0.0,
                        min_ovlp=c["min_ovlp"], reduce_mem="1g"))
    return out


def _room(c):
    """Bytes that hold the set's output.bin: at most 1.3 edges per read-end here, and the record heads."""
    return 12 * max(1, c["read_len"] - c["min_ovlp"]) + int(8 * 1.3 * 2 * c["reads"]) + (1 << 16)


def _pinned(n):
    return torch.zeros(n, dtype=torch.uint8, pin_memory=True).numpy()


# ---------------------------------------------------------------- preparing and running
class _State:
    """What the program holds for one case; jobs and servers are closed with it."""

    def __init__(self, case):
        self.case, self.jobs, self.server = case, [], None

    def __del__(self):
        if self.server is not None:
            self.server.close()
        for j in self.jobs:
            j.close()


def _new_job(c):
    return _engine().job(min_ovlp=c["min_ovlp"], reduce_mem=c["reduce_mem"])


def _feed(job, fastq):
    torch.cuda.synchronize()
    job.feed_device(fastq.data_ptr(), fastq.numel())


def prepare(case, seed):
    st = _State(case)
    kind = case["kind"]
    if kind in ("sort", "sort_static"):
        n = case["pairs"]
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        fp1 = torch.randint(0, (1 << 29) - 3, (n,), generator=gen, device="cuda")
        fp2 = torch.randint(0, (1 << 29) - 33, (n,), generator=gen, device="cuda")
        st.keys = fp1 << 32 | fp2
        # one pair in five repeats another one's fingerprint, as overlapping reads' ends do
        dup = torch.nonzero(torch.rand(n, generator=gen, device="cuda") < 0.2).view(-1)
        st.keys[dup] = st.keys[torch.randint(0, n, dup.shape, generator=gen, device="cuda")]
        # read-end ids in list order, the first half suffixes, the second prefixes (bit 31)
        st.vals = (torch.arange(n, device="cuda") % (n // 2 + 1) +
                   (torch.arange(n, device="cuda") > n // 2) * -(1 << 31)).to(torch.int32)
        st.k, st.v = torch.empty_like(st.keys), torch.empty_like(st.vals)
        st.stream = torch.cuda.Stream()
        del fp1, fp2, dup
    elif kind == "job":
        st.jobs.append(_new_job(case))
        _feed(st.jobs[0], _fastq(case, seed))
        st.out = _pinned(_room(case))
    elif kind == "host":
        st.fastq = _fastq(case, seed).cpu().numpy().tobytes()
        st.out = np.zeros(_room(case), dtype=np.uint8)
        _engine()
    elif kind == "graph":
        with _new_job(case) as job:
            _feed(job, _fastq(case, seed))
            job.run()
            st.n_reads = job.stats()["n_reads"]
            st.output = job.output()
        st.starts = np.zeros(2 * st.n_reads + 1, dtype=np.uint64)
    else:
        sets = _sets(case, seed)
        st.rooms = [_room(c) for c in sets]
        st.out = _pinned(sum(st.rooms))
        if kind == "served":
            st.fastq = []
            st.server = emp.Server(_engine())
        for k, c in enumerate(sets):
            st.jobs.append(_new_job(c))
            fq = _fastq(c, seed * 1_000_003 + k)
            if kind == "batch":
                _feed(st.jobs[-1], fq)
            else:
                st.fastq.append(_pinned(fq.numel()))
                st.fastq[-1][:] = fq.cpu().numpy()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # the engine takes its memory from a pool of its own
    return st


def run(st):
    kind = st.case["kind"]
    if kind in ("sort", "sort_static"):
        with torch.cuda.stream(st.stream):  # unsorted pairs arrive in the buffers that are sorted
            st.k.copy_(st.keys)
            st.v.copy_(st.vals)
        args = (st.k.data_ptr(), st.v.data_ptr(), st.case["pairs"], st.stream.cuda_stream)
        if kind == "sort":
            _engine().sort_pairs(*args)
        else:
            emp.sort_pairs_static(*args)
        return [st.k, st.v]
    # an output.bin ends inside the buffer that it is written to: the buffer is returned whole (zero behind it), with
    # the bytes written
    if kind == "job":
        st.jobs[0].run()
        size = st.jobs[0].output_into(st.out)
        return [st.out, size]
    if kind == "host":
        c = st.case
        out, _stats = emp.run_bytes(st.fastq, engine=_engine(), min_ovlp=c["min_ovlp"], reduce_mem=c["reduce_mem"])
        st.out[:len(out)] = np.frombuffer(out, dtype=np.uint8)
        return [st.out, len(out)]
    if kind == "graph":
        with emp.Graph(_engine(), st.output, st.n_reads) as g:
            order, starts = g.unitigs()
        st.starts[:starts.size] = starts
        return [order, st.starts, int(starts.size)]
    start = np.cumsum([0] + st.rooms)
    sizes = np.zeros(len(st.jobs), dtype=np.int64)
    if kind == "batch":
        _engine().run_batch(st.jobs)
        for i, j in enumerate(st.jobs):
            sizes[i] = j.output_into(st.out[start[i]:start[i + 1]])
        return [st.out, sizes]
    for j, fq in zip(st.jobs, st.fastq):  # served
        j.reset()
        j.feed_async(fq)
        st.server.submit(j)
    index = {id(j): i for i, j in enumerate(st.jobs)}
    waiting = len(st.jobs)
    while waiting:
        for j in st.server.step():
            i = index[id(j)]
            sizes[i] = j.output_into(st.out[start[i]:start[i + 1]])
            waiting -= 1
    return [st.out, sizes]


# ---------------------------------------------------------------- bytes that a pass cannot do without
def _fastq_bytes(c):
    n, total, lo, d = c["reads"], 0, 0, 1
    while lo < n:
        hi = min(n, 10 ** d)
        total += (hi - lo) * (7 + d + 2 * c["read_len"])
        lo, d = hi, d + 1
    return total


def _output_bytes(c):
    """Nearly one edge per distinct read-end, 8 bytes each."""
    n, g = c["reads"] * (1.0 - c["n_frac"]), max(c["genome"], 1)
    return 8 * 2 * g * (1.0 - math.exp(-n / g)) + 12 * max(0, c["read_len"] - c["min_ovlp"])


def work(case):
    kind = case["kind"]
    if kind in ("sort", "sort_static"):
        return {"bytes": 24.0 * case["pairs"], "flops": 0.0}
    if kind == "graph":  # output.bin in, the read-ends in unitig order and the unitigs' starts out
        return {"bytes": _output_bytes(case) + 8.0 * case["reads"], "flops": 0.0}
    sets = _sets(case, 0) if kind in ("batch", "served") else [case]
    return {"bytes": float(sum(_fastq_bytes(c) + _output_bytes(c) for c in sets)), "flops": 0.0}


def exact(case, seed):
    """Every output is whole numbers or bytes: there is nothing to compare in 64 bits."""
    return None
