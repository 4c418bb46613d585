"""The one-thread-per-hit DP at the edges of its blocks and of its arithmetic.

A block sorts the hits of equally long reads by the rows of their forward pass
and takes one, two or four rounds of 128 of them, by the size of the batch; its
scores are whole numbers held in floats, which bounds the length of a read
(longer ones run one hit per warp, in integers)."""
import os

import numpy as np
import pytest

import oracle as O
from clast_b200 import api, synth
from _cases import compare
from test_gpu_dp_warp import hits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap,local", [(2, 0), (4, 1), (5, 0), (8, 0), (8, 1), (9, 1), (10, 0), (16, 0)])
@pytest.mark.parametrize("reads", [1, 33, 400])
def test_equally_long_reads_equal_oracle(engine, reads, gap, local):
    rng = np.random.Generator(np.random.PCG64(reads + 7 * gap + local))
    t = synth.make_target(rng, 50_000, n_contigs=3, median=15_000, repeat_frac=0.2, n_families=3)
    q = synth.make_reads_fixed(rng, t, reads, length=97, sub=0.04, indel=0.02)
    s = api.Setting(lmer=11, stride=3, gap=gap, local=local, total_db=float(t.offsets[-1]))
    tl = api.SeqList(s.lmer).add_targets([t.seq(i).tobytes() for i in range(len(t))])
    ql = api.SeqList(s.lmer).add_queries([q.seq(i).tobytes() for i in range(len(q))])
    tbases, tgw, tln = tl.window(0, len(tl.lengths))
    qbases, qgw, qln = ql.window(0, len(ql.lengths))
    want = O.window_search(s, tbases, tgw, tln, 0, qbases, qgw, qln, 0)
    compare(hits(engine, s, tl, ql, "off"), want)


@pytest.mark.parametrize("reads", [150_000, 300_000, 600_000])
def test_blocks_of_several_rounds_match_one_hit_per_warp(engine, reads):
    """Batches of two, four and eight waves of the grid (one, two and four
    rounds per block): every field as the integer kernel gives it."""
    rng = np.random.Generator(np.random.PCG64(reads))
    t = synth.make_target(rng, 2_000_000, n_contigs=2, median=900_000)
    q = synth.make_reads_fixed(rng, t, reads, length=61)
    s = api.Setting(total_db=float(t.offsets[-1]))
    _, t_loads = api.ram_loads(np.diff(t.offsets), 64_000_000)
    _, q_loads = api.ram_loads(np.diff(q.offsets), 32_000_000)
    T = engine.targets(s, t.bases, t.offsets, t_loads, 64_000_000)
    out = {}
    for mode in ("off", "all"):
        os.environ["CLAST_DP_WARP"] = mode
        try:
            r = engine.map(s, T, q.bases, q.offsets, q_loads, 2_000_000)
        finally:
            os.environ.pop("CLAST_DP_WARP", None)
        out[mode] = {f: np.array(r[f]) for f in api.MAP_FIELDS}
        del r
    T.close()
    assert len(out["off"]["score"]) > reads // 2
    for f in api.MAP_FIELDS:
        assert np.array_equal(out["off"][f], out["all"][f]), f


@pytest.mark.parametrize("length", [(1 << 20) - 40, 1 << 20, (1 << 20) + 1])
def test_longest_reads_equal_oracle(engine, length):
    """Reads around the length above which hits run one per warp."""
    rng = np.random.Generator(np.random.PCG64(length))
    t = synth.make_target(rng, length + 3000, n_frac=0.0)
    read = t.bases[1000:1000 + length].copy()
    at = rng.integers(0, length, size=2000)
    read[at] = synth.ACGT[rng.integers(0, 4, size=2000)]
    s = api.Setting(total_db=float(t.offsets[-1]))
    tl = api.SeqList(s.lmer).add_targets([t.seq(0).tobytes()])
    ql = api.SeqList(s.lmer).add_queries([read.tobytes()])
    tbases, tgw, tln = tl.window(0, 1)
    qbases, qgw, qln = ql.window(0, 2)
    want = O.window_search(s, tbases, tgw, tln, 0, qbases, qgw, qln, 0)
    assert len(want["t_id"]) > 0 and want["score"].max() > length // 2
    compare(hits(engine, s, tl, ql, "off"), want)


@pytest.mark.parametrize("gap,local", [(4, 0), (5, 0), (5, 1), (6, 0), (7, 1), (8, 0), (8, 1), (10, 1), (14, 0), (15, 0)])
def test_bands_of_a_full_grid_match_one_hit_per_warp(engine, gap, local):
    """More equally long hits than three blocks per SM hold (bands of 5 - 8 run
    four to an SM then), and the bands next to those that take the row's letter
    pairs in another number of parts."""
    rng = np.random.Generator(np.random.PCG64(gap + 100 * local))
    t = synth.make_target(rng, 1_000_000, n_contigs=2, median=400_000)
    q = synth.make_reads_fixed(rng, t, 130_000, length=61, sub=0.04, indel=0.02)
    s = api.Setting(gap=gap, local=local, total_db=float(t.offsets[-1]))
    _, t_loads = api.ram_loads(np.diff(t.offsets), 64_000_000)
    _, q_loads = api.ram_loads(np.diff(q.offsets), 32_000_000)
    T = engine.targets(s, t.bases, t.offsets, t_loads, 64_000_000)
    out = {}
    for mode in ("off", "all"):
        os.environ["CLAST_DP_WARP"] = mode
        try:
            r = engine.map(s, T, q.bases, q.offsets, q_loads, 2_000_000)
        finally:
            os.environ.pop("CLAST_DP_WARP", None)
        out[mode] = {f: np.array(r[f]) for f in api.MAP_FIELDS}
        del r
    T.close()
    assert len(out["off"]["score"]) > 60_000
    for f in api.MAP_FIELDS:
        assert np.array_equal(out["off"][f], out["all"][f]), f
