"""The one-hit-per-warp DP across the rows at which it takes the rows' part out
of its potentials (every 4,096, counted from the band's ramp): passes that end
just before, at and after such a row, and of several of them.  One kernel runs
every hit; the oracle holds plain scores."""
import numpy as np
import pytest

import oracle as O
from clast_b200 import api, synth
from _cases import compare
from test_gpu_dp_warp import hits

pytestmark = pytest.mark.gpu

ROWS = 4096


@pytest.mark.parametrize("gap,local", [(2, 0), (8, 0), (8, 1), (16, 0), (16, 1)])
def test_passes_around_the_rebased_rows_equal_oracle(engine, gap, local):
    s = api.Setting(gap=gap, local=local)
    rng = np.random.Generator(np.random.PCG64(gap + local))
    t = synth.make_target(rng, 30_000, n_frac=0.0)
    # the read's first l-mer matches, so a pass has len - l rows; the last ones hold errors
    reads = []
    for rows in (ROWS - 1, ROWS, ROWS + gap - 1, ROWS + gap, ROWS + gap + 1, 2 * ROWS + gap, 3 * ROWS + 5):
        for flip in (False, True):
            at = int(rng.integers(100, 30_000 - 14_000))
            read = t.bases[at:at + rows + s.lmer].copy()
            for p in rng.integers(s.lmer, len(read), size=len(read) // 40):
                read[p] = synth.ACGT[rng.integers(0, 4)]
            reads.append((synth.revcomp(read) if flip else read).tobytes())
    s.total_db = float(t.offsets[-1])
    tl = api.SeqList(s.lmer).add_targets([t.seq(0).tobytes()])
    ql = api.SeqList(s.lmer).add_queries(reads)
    tb, tg, tn = tl.window(0, 1)
    qb, qg, qn = ql.window(0, len(ql.lengths))
    want = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
    assert len(want["t_id"]) >= len(reads) and want["score"].max() > 2 * ROWS
    compare(hits(engine, s, tl, ql, "all"), want)
