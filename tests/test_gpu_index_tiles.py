"""The index build at the edges of its tiles (1,024 sorted samples): sample
counts around a tile, runs of one l-mer that end at, cross or span tiles, with
and without the repeat cut, codes in one word with their position and in two."""
import numpy as np
import pytest

import oracle as O
from clast_b200 import api, synth
from _cases import compare

pytestmark = pytest.mark.gpu


def case(seed, samples, stride, lmer, poly):
    """A target of about `samples` samples with runs of poly-A, poly-AC and N,
    and reads from it and from the runs."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n = samples * stride
    parts = np.array_split(synth.ACGT[rng.integers(0, 4, size=n)], 3)
    seqs = [bytearray(p.tobytes()) for p in parts]
    if poly:
        at = len(seqs[1]) // 3
        seqs[1][at:at + poly] = b"A" * poly
        seqs[2][10:10 + poly // 2] = b"AC" * (poly // 4)
        seqs[0][-40:] = b"A" * 40  # up to the joint
        seqs[2][-30:-20] = b"N" * 10
    t = [bytes(x) for x in seqs]
    reads = []
    for s in t:
        for p in rng.integers(0, max(1, len(s) - 120), size=8):
            reads.append(s[p:p + 120])
    if poly:
        reads += [b"A" * 60 + t[0][50:90], b"AC" * 30, t[1][len(t[1]) // 3 - 50:len(t[1]) // 3 + 50]]
    return t, [r for r in reads if len(r) >= lmer]


@pytest.mark.parametrize("lmer,cut", [(8, -1), (8, 20), (15, 20), (15, 3), (15, 5000), (15, -1), (24, 20), (31, -1)])
@pytest.mark.parametrize("samples,poly", [(60, 0), (1023, 0), (1024, 0), (1025, 0), (1600, 900), (4096, 7000), (9000, 1000)])
def test_index_tiles_equal_oracle(engine, samples, poly, lmer, cut):
    stride = 3 if lmer < 24 else 2
    t, reads = case(samples + lmer, samples, stride, lmer, poly)
    s = api.Setting(lmer=lmer, stride=stride, cut_repeat=cut, total_db=float(sum(map(len, t))))
    tl = api.SeqList(s.lmer).add_targets(t)
    ql = api.SeqList(s.lmer).add_queries(reads)
    tb, tg, tn = tl.window(0, len(t))
    qb, qg, qn = ql.window(0, len(ql.lengths))
    want = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
    ix = engine.hash_table(s, tl, 0, len(t))
    compare(engine.hit_list(s, ix, ql, 0, len(reads)), want)
    ix.close()


@pytest.mark.parametrize("real", [0, 20, 150, 900, 30_000])
@pytest.mark.parametrize("cut", [-1, 3])
def test_free_records_between_few_keys(engine, real, cut):
    """A window of N's with `real` bases in it: free stretches within a tile,
    of one record to many whole chunks of 4,096, and a table without a record.
    The full index built before it leaves its records in the memory that the
    new table is given."""
    rng = np.random.Generator(np.random.PCG64(real + 10 + cut))
    n = 240_000
    t = synth.ACGT[rng.integers(0, 4, size=n)]
    s = api.Setting(lmer=12, stride=2, cut_repeat=cut, total_db=float(n))
    full = api.SeqList(s.lmer).add_targets([t.tobytes()])
    sparse_seq = np.full(n, ord("N"), np.uint8)
    at = n // 3
    sparse_seq[at:at + real] = t[at:at + real]
    sparse = api.SeqList(s.lmer).add_targets([sparse_seq.tobytes()])
    reads = [t[p:p + 100].tobytes() for p in list(rng.integers(0, n - 100, size=200)) + [at, at + max(0, real - 100)]]
    ql = api.SeqList(s.lmer).add_queries(reads)
    qb, qg, qn = ql.window(0, len(ql.lengths))
    for tl in (full, sparse, full):
        tb, tg, tn = tl.window(0, 1)
        want = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
        ix = engine.hash_table(s, tl, 0, 1)
        compare(engine.hit_list(s, ix, ql, 0, len(reads)), want)
        ix.close()


def test_window_without_a_sample_equals_oracle(engine):
    s = api.Setting(lmer=8, stride=90, total_db=20.0)
    tl = api.SeqList(s.lmer).add_targets([b"ACGTTGCAACGGTCATTGCA"])
    ql = api.SeqList(s.lmer).add_queries([b"ACGTTGCAACGGTCATTGCA"])
    tb, tg, tn = tl.window(0, 1)
    qb, qg, qn = ql.window(0, len(ql.lengths))
    want = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
    ix = engine.hash_table(s, tl, 0, 1)
    compare(engine.hit_list(s, ix, ql, 0, 1), want)
    ix.close()


# k_index_place looks at 256 samples of a run that leaves its tile, the kernel
# after it at 4,096 a step; the last size takes many thousand steps of a block
@pytest.mark.parametrize("cut", [-1, 257, 5000, 5_000_000])
@pytest.mark.parametrize("run", [255, 256, 257, 258, 256 + 4096, 256 + 4097, 30_000, 3_000_000])
def test_long_runs_equal_oracle(engine, run, cut):
    lmer, rng = 13, np.random.Generator(np.random.PCG64(run + cut))
    flank = [synth.ACGT[rng.integers(1, 4, size=m)].tobytes() for m in (1500, 700, 900)]  # no A beside the run
    poly = min(run, 1000)  # of `run` samples of poly-A, so many in a second sequence, up to its end
    rest = run - poly
    t = [flank[0] + (b"A" * (rest + lmer - 1) if rest else b"") + flank[1], flank[2] + b"A" * (poly + lmer - 1)]
    s = api.Setting(lmer=lmer, stride=1, cut_repeat=cut, total_db=float(sum(map(len, t))))
    reads = [x[p:p + 90] for x in flank for p in range(0, len(x) - 90, 61)]
    if run < 1_000_000:  # one l-mer of the run in each: as many seeds as the run has samples
        reads += [flank[2][-60:] + b"A" * lmer, b"A" * lmer + flank[1][:60]]
    tl = api.SeqList(s.lmer).add_targets(t)
    ql = api.SeqList(s.lmer).add_queries(reads)
    tb, tg, tn = tl.window(0, len(t))
    qb, qg, qn = ql.window(0, len(ql.lengths))
    want = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
    ix = engine.hash_table(s, tl, 0, len(t))
    compare(engine.hit_list(s, ix, ql, 0, len(reads)), want)
    ix.close()
