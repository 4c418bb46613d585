"""Target windows searched in groups: the seed filters' tiers, a read's hits in
one run over the group's windows, and the merge of the groups.

Reads from elements of 1 to 2,500 copies spread over five windows have seed
and hit counts on both sides of every tier's bound (8, 32, 256 and 2,048), many
equal scores among them, in one window and in several."""
import os

import numpy as np
import pytest

from _oracle_map import oracle_map
from clast_b200 import api, synth

pytestmark = pytest.mark.gpu

COPIES = (1, 3, 8, 9, 15, 31, 34, 70, 260, 2500)


def repeat_case(seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    ctg = [bytearray(synth.ACGT[rng.integers(0, 4, size=150_000)].tobytes()) for _ in range(6)]
    free = [(c, p) for c in range(6) for p in range(200, 149_000, 260)]
    free = [free[i] for i in rng.permutation(len(free))]
    reads = []
    for n in COPIES:
        element = synth.ACGT[rng.integers(0, 4, size=110)]
        for _ in range(n):
            c, p = free.pop()
            copy = element.copy()
            for at in rng.integers(0, 110, size=int(rng.integers(0, 3))):
                copy[at] = synth.ACGT[rng.integers(0, 4)]
            if rng.random() < 0.3:
                copy = synth.revcomp(copy)
            ctg[c][p:p + 110] = copy.tobytes()
        for k in range(3):
            read = element[:100 + 3 * k].copy()
            read[rng.integers(0, 100, size=2 * k)] = synth.ACGT[rng.integers(0, 4)]
            reads.append((synth.revcomp(read) if k == 1 else read).tobytes())
    order = rng.permutation(len(reads))
    return [bytes(x) for x in ctg], [reads[i] for i in order]


@pytest.mark.parametrize("cut,local", [(-1, 0), (-1, 1), (60, 0)])
def test_groups_of_windows_equal_oracle(engine, cut, local):
    tseqs, qseqs = repeat_case(11)
    s = api.Setting(cut_repeat=cut, local=local, stride=3, total_db=float(sum(map(len, tseqs))))
    t_vram, t_loads, q_loads, q_vram = 190_000, [4, 2], [17, 13], 2500
    want = oracle_map(s, tseqs, t_loads, t_vram, qseqs, q_loads, q_vram)
    assert len(want["score"]) > 1000
    t = np.frombuffer(b"".join(tseqs), np.uint8)
    toff = np.concatenate([[0], np.cumsum([len(x) for x in tseqs])]).astype(np.int64)
    q = np.frombuffer(b"".join(qseqs), np.uint8)
    qoff = np.concatenate([[0], np.cumsum([len(x) for x in qseqs])]).astype(np.int64)
    T = engine.targets(s, t, toff, t_loads, t_vram)
    try:
        for group in ("1", "2", "3", "4"):
            os.environ["CLAST_SEED_WINDOWS"] = group
            r = engine.map(s, T, q, qoff, q_loads, q_vram)
            assert np.array_equal(r["load_offsets"], want["load_offsets"]), group
            for f in api.MAP_FIELDS:
                if f == "evalue":
                    np.testing.assert_allclose(r[f], want[f], rtol=1e-12, atol=0)
                else:
                    np.testing.assert_array_equal(r[f], want[f], err_msg="%s, groups of %s" % (f, group))
            del r
    finally:
        os.environ.pop("CLAST_SEED_WINDOWS", None)
        T.close()


@pytest.mark.parametrize("reads", [3, (1 << 15) - 1, 1 << 15, (1 << 15) + 1])
def test_read_lengths_from_host_and_device(engine, reads):
    """The lengths of a large batch are looked at on the device: one longer
    read makes the batch uneven either way, and changes no other read's hits."""
    rng = np.random.Generator(np.random.PCG64(reads))
    t = synth.make_target(rng, 300_000, n_contigs=2, median=120_000)
    q = synth.make_reads_fixed(rng, t, reads, length=48, decoy_frac=0.0)
    s = api.Setting(total_db=float(t.offsets[-1]))
    long_read = t.bases[1000:1400]
    bases, off = np.concatenate([q.bases, long_read]), np.concatenate([q.offsets, [q.offsets[-1] + 400]])
    T = engine.targets(s, t.bases, t.offsets, [2], 64_000_000)
    try:
        runs = {}
        for name, args in (("even", (q.bases, q.offsets, [reads], 2_000_000)),
                           ("uneven", (bases, off, [reads + 1], 2_000_000)),
                           ("alone", (long_read, np.array([0, 400]), [1], 2_000_000))):
            r = engine.map(s, T, *args)
            runs[name] = ({f: np.array(r[f]) for f in api.MAP_FIELDS}, engine.stats())
            del r
    finally:
        T.close()
    (even, st), (both, st2), (alone, _) = runs["even"], runs["uneven"], runs["alone"]
    assert st["hits"] > 0 and len(alone["score"]) > 0
    last = both["read"] == reads
    assert last.any() and (~last).any()
    for f in api.MAP_FIELDS[1:]:
        np.testing.assert_array_equal(both[f][~last], even[f])
        np.testing.assert_array_equal(both[f][last], alone[f])
    assert st["dp_order_kind"] == 0 and st2["dp_order_kind"] == 1
