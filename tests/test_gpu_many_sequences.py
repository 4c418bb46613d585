"""Windows of about 2^20 sequences: a read's seeds are sorted as single words of
20 bits for the sequence where every window of the group has fewer, and go
through memory otherwise.  Reads from the first and the last records, with the
window alone and grouped with a small one."""
import numpy as np
import pytest

import oracle as O
from clast_b200 import api, synth

pytestmark = pytest.mark.gpu

LEN = 24


@pytest.mark.parametrize("records", [(1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_windows_around_2_to_20_sequences_equal_oracle(engine, records):
    rng = np.random.Generator(np.random.PCG64(records))
    s = api.Setting(stride=3)
    rec = synth.ACGT[rng.integers(0, 4, size=(records, LEN))]
    small = synth.ACGT[rng.integers(0, 4, size=(3, LEN))]
    small[1] = rec[-1]  # hits in both windows
    s.total_db = float(rec.size + small.size)
    picks = np.concatenate([np.arange(20), rng.integers(0, records, size=60), np.arange(records - 60, records)])
    reads = [rec[i] for i in picks] + [synth.revcomp(rec[i]) for i in picks[::3]] + list(small)
    for k in range(0, len(reads), 4):
        reads[k] = reads[k].copy()
        reads[k][int(rng.integers(0, LEN))] = ord("A")
    ql = api.SeqList(s.lmer).add_queries([r.tobytes() for r in reads])
    qb, qg, qn = ql.window(0, len(ql.lengths))
    q = np.concatenate(reads)
    qoff = np.arange(len(reads) + 1, dtype=np.int64) * LEN

    def window(x):  # every sequence followed by its first l - 1 bases
        n = len(x)
        return np.concatenate([x, x[:, :s.lmer - 1]], 1).tobytes(), \
            np.arange(n, dtype=np.int32) * (LEN + s.lmer - 1), np.full(n, LEN, np.int32)

    for sets in ([rec], [rec, small], [small, rec]):
        rows = []
        for load, x in enumerate(sets):
            tb, tg, tn = window(x)
            h = O.window_search(s, tb, tg, tn, 0, qb, qg, qn, 0)
            rows += [(int(h["q_id"][i]) // 2, int(h["q_id"][i]) & 1, load, int(h["t_id"][i]), int(h["t_idx"][i]),
                      int(h["q_idx"][i]), int(h["t_len"][i]), int(h["q_len"][i]), int(h["match"][i]),
                      int(h["score"][i]), float(h["evalue"][i])) for i in range(len(h["t_id"]))]
        rows.sort(key=lambda r: (r[0], -r[9]))  # stable
        assert len(rows) > len(picks) and max(r[3] for r in rows) == records - 1
        t = np.concatenate(sets).reshape(-1)
        toff = np.arange(len(t) // LEN + 1, dtype=np.int64) * LEN
        T = engine.targets(s, t, toff, [len(x) for x in sets], 64_000_000)
        r = engine.map(s, T, q, qoff, [len(reads)], 2_000_000)
        for f, want in zip(api.MAP_FIELDS, zip(*rows)):
            if f == "evalue":
                np.testing.assert_allclose(r[f], want, rtol=1e-12, atol=0)
            else:
                np.testing.assert_array_equal(r[f], want, err_msg=f)
        del r
        T.close()
