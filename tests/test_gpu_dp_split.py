"""Which hits run one per warp: the longest of an uneven batch, all equal ones of
a small batch with a wide band, none with a narrow one, as they were measured to be
faster on the B200 in either mode.  Results are the same either way."""
import os

import numpy as np
import pytest

from clast_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap,local,reads,uneven,runs", [
    (3, 1, 4000, True, "some"), (2, 0, 4000, True, "some"), (8, 1, 4000, True, "some"), (8, 0, 4000, True, "some"),
    (9, 1, 3200, False, "all"), (16, 1, 3200, False, "all"), (11, 0, 3200, False, "all"), (3, 0, 3200, False, "none"),
    (2, 1, 3200, False, "none")])
def test_split_by_band_and_mode(engine, gap, local, reads, uneven, runs):
    rng = np.random.Generator(np.random.PCG64(gap + 50 * local))
    t = synth.make_target(rng, 2_000_000, n_contigs=2, median=900_000)
    if uneven:
        q = synth.make_reads_var(rng, t, reads, len_range=(100, 5000))
    else:
        q = synth.make_reads_fixed(rng, t, reads, length=150)
    s = api.Setting(gap=gap, local=local, total_db=float(t.offsets[-1]))
    _, q_loads = api.ram_loads(np.diff(q.offsets), 32_000_000)
    T = engine.targets(s, t.bases, t.offsets, [len(t)], 64_000_000)
    out = {}
    try:
        for mode in (None, "off"):
            if mode:
                os.environ["CLAST_DP_WARP"] = mode
            r = engine.map(s, T, q.bases, q.offsets, q_loads, 2_000_000)
            st = engine.stats()
            out[mode] = {f: np.array(r[f]) for f in api.MAP_FIELDS}, st["dp_warp_hits"], st["hits"]
            del r
    finally:
        os.environ.pop("CLAST_DP_WARP", None)
        T.close()
    assert out["off"][1] == 0 and out[None][2] > 2000
    warp, total = out[None][1:]
    assert {"none": warp == 0, "some": 0 < warp < total, "all": warp == total}[runs], (warp, total)
    for f in api.MAP_FIELDS:
        np.testing.assert_array_equal(out[None][0][f], out["off"][0][f], err_msg=f)
