"""The integer DP's potentials at rows that no GPU test can reach.

The one-hit-per-warp kernel holds scores as S + 4 (row + 1) + 2 column in 32-bit
integers.  A matching read's potentials rise by 5 per row, so without taking
the rows' part out from time to time they pass 2^31 at row 429,496,729, well
below the longest read that is accepted (2^31 bases).  Here the kernel's
recurrence runs over 400 matching rows that end there, with its constants read
from its source; test_gpu_dp_rebase.py runs the kernel across the same steps at
lengths a test can afford."""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "clast_b200", "csrc",
                   "clast_kernels.cu")
OPEN, EXT, MARGIN, STEP_ROW, STEP_COL = -5, -2, -30000, 4, 2


def rebase_rows():
    m = re.search(r"constexpr int kDpRebaseRows = (\d+);", open(SRC).read())
    return int(m.group(1)) if m else None


def wrap(x):
    return (x + 2**31) % 2**32 - 2**31


def potentials(first, rows, gap, state, rebase):
    """`rows` matching rows from row `first` on in wrapping 32-bit integers;
    state: scores and vertical states per column (plain scores).  Returns the
    last row's scores as the kernel takes them out."""
    W = 2 * gap + 1
    c = np.arange(W)
    # what the kernel has taken out before row `first` (it starts one step below zero)
    out = STEP_ROW * rebase * (1 + first // rebase) if rebase else 0
    s = wrap(state[0] + STEP_ROW * first + STEP_COL * c - out)
    u = wrap(state[1] + STEP_ROW * first + STEP_COL * c - out)
    for r in range(first, first + rows):
        if rebase and r > first and r % rebase == 0:
            d = STEP_ROW * rebase
            out += d
            s, u = wrap(s - d), wrap(u - d)
        lift = STEP_ROW * (r + 1) - out
        vbot = wrap((gap + 1) * EXT + OPEN + OPEN + EXT + STEP_COL * 2 * gap + lift)
        h = wrap(MARGIN + EXT + lift)
        ns, nu = s.copy(), u.copy()
        for x in range(W):
            v = u[x + 1] if x + 1 < W else vbot
            point = 1 if x == gap else -3  # the read matches the target along the middle column
            p = max(wrap(s[x] + point + STEP_ROW), v)
            ns[x] = max(p, h)
            nu[x] = max(wrap(ns[x] + OPEN + EXT + STEP_COL), v)
            h = max(wrap(p + OPEN + EXT + STEP_COL), h)
        s, u = ns, nu
    return wrap(s - (STEP_ROW * (first + rows) - out) - STEP_COL * c)


def start_state(gap):
    c = np.arange(2 * gap + 1)
    s = np.where(c < gap, MARGIN, np.where(c == gap, 0, (c - gap) * EXT + OPEN)).astype(np.int64)
    return s, np.where(c < gap, s, s + OPEN + EXT + STEP_COL)


def steady_state(gap, rows):
    """Scores after `rows` matching rows: the middle column holds rows, its
    neighbours what opening and extending a gap from it costs."""
    c = np.arange(2 * gap + 1)
    d = np.abs(c - gap)
    s = rows - np.where(d > 0, -OPEN - EXT * d, 0) - np.where(c > gap, d, 0)
    return s.astype(np.int64), (s + OPEN + EXT + STEP_COL).astype(np.int64)


@pytest.mark.parametrize("gap", [2, 8, 16])
@pytest.mark.parametrize("last", [1000, 429_497_000, 2**30, 2**31 - 1000])
def test_matching_rows_score_their_number(gap, last):
    rebase = rebase_rows()
    first = last - 400
    state = start_state(gap) if first < 1000 else steady_state(gap, first)
    if first < 1000:
        got = potentials(0, last, gap, state, rebase)
    else:
        got = potentials(first, 400, gap, state, rebase)
    assert got[gap] == got.max() == last


def test_potentials_fit_32_bits():
    """The largest accepted score plus what the kernel leaves in a potential:
    the rows since the last step, the ramp in and out of the band, the column."""
    assert rebase_rows() is not None
    gap = 16
    left_in = STEP_ROW * 2 * (gap + 1) + STEP_COL * (2 * gap + 1)
    assert 2**31 - 1 - 300 + left_in < 2**31
    assert MARGIN - 2 * STEP_ROW * rebase_rows() > -2**31
