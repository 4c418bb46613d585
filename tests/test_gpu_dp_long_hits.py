"""One read too long for the one-per-thread DP (2^20 rows) in a batch of short
ones: its hits run one per warp, the others as in a batch without it."""
import os

import numpy as np
import pytest

import oracle as O
from clast_b200 import api, synth
from _cases import compare
from test_gpu_dp_warp import hits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("local", [0, 1])
def test_one_long_read_among_short_ones(engine, local):
    rng = np.random.Generator(np.random.PCG64(20 + local))
    rows = 1 << 20
    s = api.Setting(local=local)
    t = synth.make_target(rng, rows + 5000, n_frac=0.0)
    read = t.bases[2000:2000 + rows + s.lmer + 9].copy()
    at = rng.integers(s.lmer, len(read), size=3000)
    read[at] = synth.ACGT[rng.integers(0, 4, size=3000)]
    below = t.bases[1000:1000 + rows + s.lmer - 1].copy()  # one row less than the bound
    at = rng.integers(s.lmer, len(below), size=3000)
    below[at] = synth.ACGT[rng.integers(0, 4, size=3000)]
    q = synth.make_reads_var(rng, t, 4000, len_range=(100, 200))
    s.total_db = float(t.offsets[-1])
    short = [q.seq(i).tobytes() for i in range(len(q))]
    tl = api.SeqList(s.lmer).add_targets([t.seq(0).tobytes()])
    ql = api.SeqList(s.lmer).add_queries(short[:2000] + [read.tobytes(), below.tobytes()] + short[2000:])
    tb, tg, tn = tl.window(0, 1)
    qb, qg, qn = ql.window(0, len(ql.lengths))
    want = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
    assert len(want["t_id"]) > 3000 and want["score"].max() > rows // 2
    seeds = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0, stage=O.STAGE_FILTERED)
    long_hits = int((qn[seeds["q_id"]] - s.lmer >= rows).sum())
    assert 0 < long_hits < 1000
    for mode in ("off", None, "all"):
        before = engine.stats()
        compare(hits(engine, s, tl, ql, mode), want)
        after = engine.stats()
        warp, total = (after[k] - before[k] for k in ("dp_warp_hits", "hits"))
        assert total == len(seeds["t_id"])
        if mode == "off":
            assert warp == long_hits
        elif mode is None:
            assert long_hits <= warp < total
        else:
            assert warp == total
