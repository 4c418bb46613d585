"""Seeding of whole reads at its tiers' bounds: reads of one, three and more
rounds of 160 l-mers, slots of up to 8, 16, 32 and more seeds, 32-bit and 64-bit
l-mers, one to four windows per group, non-ACGT bases and palindromes."""
import os

import numpy as np
import pytest

from _oracle_map import oracle_map
from clast_b200 import api, synth

pytestmark = pytest.mark.gpu


def case(seed, lmer):
    rng = np.random.Generator(np.random.PCG64(seed))
    t = synth.make_target(rng, 240_000, n_contigs=6, median=35_000, repeat_frac=0.3, n_families=4, fam_len=(200, 900))
    tseqs = [bytearray(t.seq(i).tobytes()) for i in range(len(t))]
    comp = bytes.maketrans(b"ACGT", b"TGCA")
    for s in tseqs:  # l-mers that are their own reverse complement, and an AT run (many of them)
        for p in range(500, len(s) - 400, 9000):
            half = bytes(s[p:p + 40])
            s[p + 40:p + 80] = half.translate(comp)[::-1]
            s[p + 200:p + 260] = b"AT" * 30
    reads = []
    lens = [lmer - 1, lmer, lmer + 1, 159 + lmer, 160 + lmer, 161 + lmer, 479 + lmer, 480 + lmer, 481 + lmer, 1500, 60, 100, 150]
    for n in lens:
        for _ in range(4):
            s = tseqs[int(rng.integers(0, len(tseqs)))]
            if len(s) <= n + 1:
                continue
            p = int(rng.integers(0, len(s) - n))
            r = bytearray(s[p:p + n])
            for at in rng.integers(0, max(1, n), size=n // 60):
                r[at] = b"ACGTN"[int(rng.integers(0, 5))]
            reads.append(bytes(r) if rng.random() < 0.5 else bytes(r).translate(comp)[::-1])
    for s in tseqs:
        reads.append(bytes(s[480:640]))
        reads.append(bytes(s[690:780]))
    return [bytes(x) for x in tseqs], reads


@pytest.mark.parametrize("lmer,stride", [(8, 2), (12, 3), (15, 5), (16, 4), (17, 4), (24, 3), (31, 2)])
@pytest.mark.parametrize("local", [0, 1])
def test_reads_of_every_tier_equal_oracle(engine, lmer, stride, local):
    tseqs, reads = case(100 + lmer, lmer)
    s = api.Setting(lmer=lmer, stride=stride, local=local, total_db=float(sum(map(len, tseqs))))
    t_loads, t_vram, q_loads, q_vram = [len(tseqs)], 70_000, [20, len(reads) - 20], 9000
    want = oracle_map(s, tseqs, t_loads, t_vram, reads, q_loads, q_vram)
    assert len(want["score"]) > 30
    t = np.frombuffer(b"".join(tseqs), np.uint8)
    toff = np.concatenate([[0], np.cumsum([len(x) for x in tseqs])]).astype(np.int64)
    q = np.frombuffer(b"".join(reads), np.uint8)
    qoff = np.concatenate([[0], np.cumsum([len(x) for x in reads])]).astype(np.int64)
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
