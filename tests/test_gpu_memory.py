"""Maps that run short of device memory: a group of windows is searched at once
when its hits fit, else window by window.  And the pinned memory that calls keep."""
import os

import numpy as np
import pytest

from clast_b200 import api, synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


class Hold:
    """Device memory taken until a given amount is free."""

    def __init__(self):
        import torch
        self.torch, self.blocks = torch, []

    def leave(self, free):
        self.blocks = []
        self.torch.cuda.empty_cache()
        self.torch.cuda.synchronize()
        for unit in (16 << 30, 1 << 30, 64 * MB, 2 * MB):
            while self.torch.cuda.mem_get_info()[0] - unit >= free:
                try:
                    self.blocks.append(self.torch.empty(unit, dtype=self.torch.uint8, device="cuda"))
                except self.torch.cuda.OutOfMemoryError:  # no stretch of that size is left
                    break

    def close(self):
        self.blocks = []
        self.torch.cuda.empty_cache()


def repeats(n_reads):
    """Two contigs of 1 Mbp holding 20 copies each of one 20 kbp stretch, and reads from it."""
    rng = np.random.Generator(np.random.PCG64(77))
    element = synth.ACGT[rng.integers(0, 4, size=20_000)]
    ctg = []
    for _ in range(2):
        c = synth.ACGT[rng.integers(0, 4, size=1_000_000)].copy()
        for k in range(20):
            c[k * 50_000 + 100:k * 50_000 + 20_100] = element
        ctg.append(c)
    at = rng.integers(0, 20_000 - 100, size=n_reads)
    reads = element[at[:, None] + np.arange(100)]
    return np.concatenate(ctg), np.array([0, 1_000_000, 2_000_000], np.int64), np.ascontiguousarray(reads).reshape(-1), \
        np.arange(n_reads + 1, dtype=np.int64) * 100


def test_group_that_does_not_fit_is_searched_window_by_window():
    t, toff, q, qoff = repeats(60_000)
    n = len(qoff) - 1
    s = api.Setting(cut_repeat=-1, total_db=float(len(t)))
    eng, hold = api.Engine(0), Hold()
    T = eng.targets(s, t, toff, [2], 1_000_100)  # a window per contig

    def run(group=None):
        eng.trim()
        if group:
            os.environ["CLAST_SEED_WINDOWS"] = group
        try:
            r = eng.map(s, T, q, qoff, [n], 2_000_000)
        finally:
            os.environ.pop("CLAST_SEED_WINDOWS", None)
        out = {f: np.array(r[f]) for f in api.MAP_FIELDS}
        del r
        return out, eng.stats()

    try:
        want, ample = run()
        assert ample["hits"] > 2_000_000  # some 85 bytes each, with the windows' together
        free = 128 * MB
        while True:  # what one window at a time needs
            eng.trim()
            hold.leave(free)
            try:
                run("1")
                break
            except api.ClastError as e:
                assert e.code == -3, str(e)
                free += 32 * MB
                assert free < 4096 * MB
        eng.trim()
        hold.leave(free + 48 * MB)
        got, short = run()
        for f in api.MAP_FIELDS:
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
        # it did not fit at once, and what it counted before that is not counted twice
        assert short["map_launches"] > ample["map_launches"]
        for k in ("seeds", "hits", "dp_cells", "query_kmers"):
            assert short[k] == ample[k], k
    finally:
        hold.close()
        T.close()
        eng.close()


def pinned():
    """Bytes of pinned host memory of this process (the runtime maps it from /dev/zero)."""
    total = 0
    for line in open("/proc/self/maps"):
        x = line.split()
        if len(x) > 5 and x[5] == "/dev/zero":
            a, b = x[0].split("-")
            total += int(b, 16) - int(a, 16)
    return total


def test_pinned_staging_is_bounded_and_trimmed():
    """Offsets that do not start at 0 are made relative on the host: 32 MB of them
    must not stay pinned (16 MB may, until clast_ctx_trim)."""
    n = 4_000_000
    rng = np.random.Generator(np.random.PCG64(5))
    t = synth.make_target(rng, 200_000, n_contigs=2, median=90_000)
    q = synth.ACGT[rng.integers(0, 4, size=20 * (n + 1))]
    qoff = np.arange(n + 2, dtype=np.int64) * 20
    s = api.Setting(total_db=float(t.offsets[-1]))
    eng = api.Engine(0)
    T = eng.targets(s, t.bases, t.offsets, [2], 64_000_000)
    try:
        for off in (qoff[:-1], qoff[:-1], qoff[1:]):  # the same sizes everywhere else: only the last one shifts
            before = pinned()
            r = eng.map(s, T, q, off, [n], 2_000_000)
            del r
            grown = pinned() - before
        assert before > 0
        assert grown < 20 * MB, grown
        eng.trim()
        kept = pinned()
        r = eng.map(s, T, q, qoff[1:1_500_002], [1_500_000], 2_000_000)  # 12 MB: staged
        del r
        assert pinned() - kept >= 12 * MB
        eng.trim()
        assert pinned() == kept
    finally:
        T.close()
        eng.close()


def test_failed_builds_leave_the_context_usable():
    """Targets whose later windows find no memory while the earlier ones are being
    indexed: the call fails, and the next ones are not disturbed by what was queued."""
    rng = np.random.Generator(np.random.PCG64(6))
    t = synth.make_target(rng, 32_000_000, n_contigs=8, median=4_000_000)
    q = synth.make_reads_fixed(rng, t, 3000, length=120)
    small = synth.make_target(rng, 1_000_000, n_contigs=2, median=400_000)
    qs = synth.make_reads_fixed(rng, small, 2000, length=120)
    s = api.Setting(total_db=float(t.offsets[-1]))
    eng, hold = api.Engine(0), Hold()

    def mapped(target, reads, t_vram):
        T = eng.targets(s, target.bases, target.offsets, [len(target)], t_vram)
        r = eng.map(s, T, reads.bases, reads.offsets, [len(reads)], 2_000_000)
        out = {f: np.array(r[f]) for f in api.MAP_FIELDS}
        del r
        T.close()
        return out

    try:
        want, want_small = mapped(t, q, 4_500_000), mapped(small, qs, 64_000_000)
        failed = 0
        for free in (256 * MB, 320 * MB, 384 * MB):
            eng.trim()
            hold.leave(free)
            try:
                mapped(t, q, 4_500_000)
            except api.ClastError as e:
                assert e.code == -3, str(e)
                failed += 1
            got = mapped(small, qs, 64_000_000)  # at once, in what the failed call gave back
            for f in api.MAP_FIELDS:
                np.testing.assert_array_equal(got[f], want_small[f], err_msg=f)
        assert failed > 0
        hold.close()
        got = mapped(t, q, 4_500_000)
        for f in api.MAP_FIELDS:
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
    finally:
        hold.close()
        eng.close()


def test_released_results_make_room_for_the_next():
    """Maps in a loop, each result released before the next: the device never holds
    two of them."""
    from cuda.bindings import runtime as rt
    from cuda.bindings.driver import cuuint64_t
    rng = np.random.Generator(np.random.PCG64(8))
    t = synth.make_target(rng, 4_000_000, n_contigs=4, median=900_000)
    q = synth.make_reads_fixed(rng, t, 400_000, length=60)
    s = api.Setting(total_db=float(t.offsets[-1]))
    _, q_loads = api.ram_loads(np.diff(q.offsets), 32_000_000)
    attr = rt.cudaMemPoolAttr
    eng = api.Engine(0)
    _, pool = rt.cudaDeviceGetDefaultMemPool(0)

    def mb(a):
        return int(rt.cudaMemPoolGetAttribute(pool, a)[1]) / MB

    high = []
    try:
        eng.trim()
        for _ in range(5):
            rt.cudaMemPoolSetAttribute(pool, attr.cudaMemPoolAttrUsedMemHigh, cuuint64_t(0))
            T = eng.targets(s, t.bases, t.offsets, [len(t)], 64_000_000)
            r = eng.map(s, T, q.bases, q.offsets, q_loads, 2_000_000)
            slab = 48 * len(r["read"]) / MB
            del r
            T.close()
            high.append(mb(attr.cudaMemPoolAttrUsedMemHigh))
    finally:
        eng.close()
    assert slab > 10
    assert max(high) - high[0] < slab / 2, (high, slab)
