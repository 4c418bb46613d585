"""Few reads with many seeds each: their seed partitions overflow, the search runs
again with larger ones, and the next such search starts with those."""
import numpy as np
import pytest

from _oracle_map import oracle_map
from clast_b200 import api, synth

pytestmark = pytest.mark.gpu


def test_partitions_that_overflowed_are_remembered():
    rng = np.random.Generator(np.random.PCG64(4))
    element = synth.ACGT[rng.integers(0, 4, size=160)]
    half = [np.concatenate([x for _ in range(350) for x in (element, synth.ACGT[rng.integers(0, 4, size=40)])])
            for _ in range(2)]
    reads = []
    for k in range(100):
        r = element[:150].copy()
        r[rng.integers(0, 150, size=2)] = synth.ACGT[rng.integers(0, 4, size=2)]
        reads.append(r)
    t, toff = np.concatenate(half), np.array([0, len(half[0]), len(half[0]) + len(half[1])], np.int64)
    q, qoff = np.concatenate(reads), np.arange(101, dtype=np.int64) * 150
    s = api.Setting(cut_repeat=-1, width=30, total_db=float(len(t)))
    t_vram = len(half[0]) + 1000  # a window per half
    want = oracle_map(s, [x.tobytes() for x in half], [2], t_vram, [r.tobytes() for r in reads], [100], 2_000_000)
    assert len(want["score"]) >= 100
    eng = api.Engine(0)
    launches = []
    try:
        T = eng.targets(s, t, toff, [2], t_vram)
        for _ in range(3):
            r = eng.map(s, T, q, qoff, [100], 2_000_000)
            for f in api.MAP_FIELDS:
                if f == "evalue":
                    np.testing.assert_allclose(r[f], want[f], rtol=1e-12, atol=0)
                else:
                    np.testing.assert_array_equal(r[f], want[f], err_msg=f)
            del r
            st = eng.stats()
            launches.append(st["map_launches"])
        T.close()
    finally:
        eng.close()
    assert st["seeds"] > 1_000_000
    assert launches[1] < launches[0] and launches[2] == launches[1], launches
