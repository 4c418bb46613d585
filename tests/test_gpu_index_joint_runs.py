"""Runs of one l-mer whose samples lie on joints, with the repeat cut off or
large: many short records that share their ends.  Such a run spans many tiles
of the index build and keeps no sample, one, or a few in its last tiles."""
import numpy as np
import pytest

import oracle as O
from clast_b200 import api, synth
from _cases import compare

pytestmark = pytest.mark.gpu


def joint_run(lmer, records, tail, seed):
    """A contig, `records` records of lmer - 1 A's (every sample of them on a
    joint) and a contig that holds `tail` more A's than those samples need:
    tail - lmer + 1 kept ones at the run's end.  Reads from the contigs and
    across the A's."""
    rng = np.random.Generator(np.random.PCG64(seed))
    flank = [synth.ACGT[rng.integers(1, 4, size=m)].tobytes() for m in (1500, 40, 1400)]  # no A in them
    t = [flank[0]] + [b"A" * (lmer - 1)] * records + [flank[1] + b"A" * tail + flank[2]]
    reads = [x[p:p + 90] for x in (flank[0], flank[2]) for p in range(0, len(x) - 90, 61)]
    if tail:
        reads += [flank[1] + b"A" * tail + flank[2][:60]]
    return t, reads


@pytest.mark.parametrize("lmer,records,cut,tail", [
    (15, 200_000, -1, 0), (15, 200_000, -1, 1), (15, 200_000, 50_000_000, 40), (31, 80_000, -1, 1),
    (15, 50_000, 5000, 40), (15, 3000, -1, 0), (15, 3000, -1, 1), (31, 3000, 1_000_000, 40), (15, 100, -1, 40),
    (15, 100, 300, 1), (31, 20, -1, 1)])
def test_runs_on_joints_equal_oracle(engine, lmer, records, cut, tail):
    tail = tail + lmer - 1 if tail else 0
    t, reads = joint_run(lmer, records, tail, records + tail + lmer)
    s = api.Setting(lmer=lmer, stride=1, cut_repeat=cut, total_db=float(sum(map(len, t))))
    tl = api.SeqList(s.lmer).add_targets(t)
    ql = api.SeqList(s.lmer).add_queries(reads)
    tb, tg, tn = tl.window(0, len(t))
    qb, qg, qn = ql.window(0, len(ql.lengths))
    want = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
    assert len(want["t_id"]) >= len(reads) - 2
    ix = engine.hash_table(s, tl, 0, len(t))
    compare(engine.hit_list(s, ix, ql, 0, len(reads)), want)
    ix.close()
