"""Timed cases of the search path: what a user of the library has it do.

Every case is one pass through the public entry points (clast_b200.api):

* ``map``    -- reads against targets whose index is resident (Engine.map), as
  a program does that keeps one genome and is handed read sets;
* ``job``    -- a whole job: index the targets, map the reads (Engine.targets
  then Engine.map), as the command line does for one pair of files;
* ``text``   -- ``map`` and the 10-column text of its result (Engine.format_tsv_text);
* ``window`` -- one query window against one resident window index through the
  per-window seam (Engine.hit_list_window);
* ``served`` -- a burst of requests to a Server, submitted together, each polled.

Inputs are synthetic DNA of the shapes of clast_b200/synth.py, drawn on the GPU
from the seed: contigs of uniform bases with repeat families (copies of 300 bp
- 6 kbp at 80-99 % identity) and short N runs; reads with substitutions, indels,
both strands and random decoys.

How many hits a pass gives depends on the inputs.  So that outputs of one case
always have one shape, they come in two parts: the first ``head`` hits as the
library's own arrays, and the others in arrays of ``tail`` hits, zeros after them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from clast_b200 import api

T_RAM, Q_RAM, Q_VRAM = 64_000_000, 32_000_000, 2_000_000  # the command line's defaults (64 MBase; reads: both strands)

_BASE = dict(kind="map", target_bp=100_000_000, contigs=200, repeats=0.10, families=500, t_vram=T_RAM, reads=1000,
             len_lo=150, len_hi=150, error="short", where="host", lmer=15, stride=5, gap=8, local=0, requests=0,
             head=0, tail=4096)


def _case(name, **kw):
    return dict(_BASE, name=name, **kw)


def listed():
    return [
        # the smallest call: one short read from host memory against a resident genome
        _case("one_read", reads=1),
        # a service's queue: requests of 1-1,000 uneven reads that arrive together
        _case("served_burst", kind="served", requests=24, reads=1000, len_lo=100, len_hi=5000, tail=120_000),
        # the largest served request in one call
        _case("large_request", reads=10_000, len_lo=100, len_hi=5000, head=35_000, tail=15_000),
        # a bacterial-size job from host memory: index and map (the repository's small workload)
        _case("small_job", kind="job", target_bp=1_000_000, contigs=1, repeats=0.0, families=0, reads=1000),
        # the repository's headline workload: index 100 Mbp and map 1,000,000 reads, inputs in HBM
        _case("medium_job", kind="job", reads=1_000_000, where="device", head=1_850_000, tail=500_000),
        # reads from pinned host memory to the result text
        _case("result_text", kind="text", reads=200_000, where="pinned", head=370_000, tail=90_000),
        # long noisy reads of very different lengths (the repository's uneven workload, a tenth of it)
        _case("uneven_reads", reads=20_000, len_lo=50, len_hi=10_000, error="noisy", where="device",
              head=100_000, tail=25_000),
        # local alignment (-local) of short reads
        _case("local_reads", reads=200_000, local=1, where="pinned", head=410_000, tail=100_000),
        # longer seeds, a sparse index and the widest band: l-mers of more than 32 bits
        _case("wide_band", reads=60_000, len_lo=300, len_hi=300, lmer=20, stride=10, gap=16, where="device",
              head=90_000, tail=20_000),
        # one large repeat-rich chromosome as a single window: many hits per read
        _case("repeat_genome", target_bp=250_000_000, contigs=1, repeats=0.45, families=1000, t_vram=260_000_000,
              reads=100_000, where="device", head=1_450_000, tail=400_000),
        # a new large chromosome and its first reads: the index build dominates
        _case("new_genome", kind="job", target_bp=250_000_000, contigs=1, repeats=0.45, families=1000,
              t_vram=260_000_000, reads=2000, where="device", head=28_000, tail=20_000),
        # the reference's own unit of work: one 2 MBase query window against one target window
        _case("query_window", kind="window", target_bp=60_000_000, contigs=100, families=300, reads=6000,
              tail=30_000),
    ]


def _copies(c):
    """Expected copies of a read's place in the target."""
    return c["repeats"] * c["repeats"] * c["target_bp"] / (c["families"] * 1900.0) if c["families"] else 0.0


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    c = dict(_BASE)
    c["kind"] = rng.choice(["map", "map", "map", "job", "text", "window", "served"])
    c["target_bp"] = _log_int(rng, 500_000, 60_000_000 if c["kind"] == "window" else 120_000_000)
    c["contigs"] = 1 if c["target_bp"] < 2_000_000 else rng.choice([1, 7, 50, 200])
    if c["contigs"] == 1:
        c["t_vram"] = 260_000_000
    c["repeats"], c["families"] = rng.choice([(0.0, 0), (0.10, max(1, c["target_bp"] // 200_000)),
                                              (0.45, max(1, c["target_bp"] // 250_000))])
    c["lmer"], c["stride"] = rng.choice([(15, 5), (15, 5), (13, 7), (16, 3), (17, 5), (24, 8)])
    c["gap"] = rng.choice([8, 8, 8, 4, 11, 16])
    c["local"] = rng.choice([0, 0, 0, 1])
    c["where"] = rng.choice(["host", "pinned", "device"])
    shape = rng.choice(["short", "short", "any", "long"])
    if shape == "long":
        c["len_lo"], c["len_hi"], c["error"] = 50, rng.choice([3000, 10_000]), rng.choice(["short", "noisy"])
    else:
        c["len_lo"] = _log_int(rng, 50, 400)
        c["len_hi"] = c["len_lo"] if shape == "short" else c["len_lo"] + rng.randrange(1, 700)
    mean = (c["len_lo"] + c["len_hi"]) / 2 if shape != "long" else c["len_hi"] / 4
    most = 12_000_000 if c["repeats"] > 0.2 or shape == "long" else 40_000_000  # bases of a pass
    if c["gap"] > 8 or c["lmer"] < 15:
        most //= 3
    if c["kind"] == "window":
        most = 900_000
    c["reads"] = _log_int(rng, 1, max(2, most / mean))
    if c["kind"] == "served":
        c["requests"] = rng.randrange(1, 33)
        c["reads"] = max(1, min(1000, c["reads"] // c["requests"]))
        c["where"] = "host"
    if c["kind"] == "window":
        c["where"] = "host"
    per_read = (4 + 3 * _copies(c)) * max(1.0, mean / 400)
    c["tail"] = int(4096 + max(1, c["requests"]) * c["reads"] * per_read)
    return c


# ---------------------------------------------------------------- inputs

_ACGT = (65, 67, 71, 84)


def _tools(seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return dev, torch.Generator(device=dev).manual_seed(int(seed)), np.random.default_rng(int(seed))


def _acgt(codes):
    return torch.tensor(_ACGT, dtype=torch.uint8, device=codes.device)[codes.long()]


def _random_bases(n, g, dev):
    return _acgt(torch.randint(0, 4, (n,), generator=g, device=dev, dtype=torch.uint8))


def _target(c, g, rs, dev):
    """(bases, offsets): contigs of log-normal length with repeat families and N runs."""
    n, k = c["target_bp"], c["contigs"]
    w = rs.lognormal(0.0, 0.9, k) if k > 1 else np.ones(1)
    floor = min(24_000, n // (2 * k))
    lens = floor + ((w / w.sum()) * (n - floor * k)).astype(np.int64)
    lens[-1] += n - lens.sum()
    b = _random_bases(n, g, dev)
    if c["families"] > 0:
        flen = np.exp(rs.uniform(math.log(300), math.log(6000), c["families"])).astype(np.int64)
        copies = np.maximum(2, (c["repeats"] * n / c["families"] / flen).astype(np.int64))
        fam = rs.permutation(np.repeat(np.arange(c["families"]), copies))
        # copies at random distances, in random order, without overlap
        gaps = rs.exponential(1.0, len(fam) + 1)
        room = n - int(flen[fam].sum())
        if room > 0:
            start = (np.cumsum(gaps)[:-1] / gaps.sum() * room).astype(np.int64) + np.cumsum(flen[fam]) - flen[fam]
            cons = _random_bases(int(flen.sum()), g, dev)
            first = np.cumsum(flen) - flen
            ln = torch.from_numpy(flen[fam]).to(dev)
            within = torch.arange(int(ln.sum()), device=dev) - torch.repeat_interleave(torch.cumsum(ln, 0) - ln, ln)
            copy = cons[torch.repeat_interleave(torch.from_numpy(first[fam]).to(dev), ln) + within]
            ident = rs.uniform(0.80 if c["repeats"] > 0.2 else 0.85, 0.99, len(fam))
            ident = torch.repeat_interleave(torch.from_numpy(ident).to(dev), ln)
            mut = torch.rand(len(copy), generator=g, device=dev, dtype=torch.float64) > ident
            copy = torch.where(mut, _random_bases(len(copy), g, dev), copy)
            b[torch.repeat_interleave(torch.from_numpy(start).to(dev), ln) + within] = copy
    for s, r in zip(rs.integers(0, n, max(1, n // 100_000)), rs.geometric(0.01, max(1, n // 100_000))):
        b[int(s):int(s + r)] = 78  # N
    return b, np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)


def _reads(c, n, tb, toff, g, rs, dev):
    """(bases, offsets) of n reads sampled from the target."""
    lens = np.exp(rs.uniform(math.log(c["len_lo"]), math.log(c["len_hi"] + 1), n)).astype(np.int64)
    lens = np.clip(lens, c["len_lo"], c["len_hi"])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    tl = np.diff(toff)
    ctg = rs.choice(len(tl), n, p=tl / tl.sum())
    span = np.maximum(1, tl[ctg] - lens)
    start = toff[ctg] + (rs.random(n) * span).astype(np.int64)
    err = rs.uniform(0.01, 0.12, n) if c["error"] == "noisy" else np.full(n, np.nan)
    sub = np.where(np.isnan(err), 0.02, 0.7 * err)
    indel = np.where(np.isnan(err), 0.005, 0.15 * err)

    def up(x):
        return torch.from_numpy(np.ascontiguousarray(x)).to(dev)

    ln, first = up(lens), up(off[:-1])
    tot = int(off[-1])
    rid = torch.repeat_interleave(torch.arange(n, device=dev), ln)
    k = torch.arange(tot, device=dev) - first[rid]

    def rand():
        return torch.rand(tot, generator=g, device=dev)

    half = up(indel / 2)[rid].float()
    ins = rand() < half
    ins[1:] |= ins[:-1] & (rand()[1:] < 0.5)
    gone = torch.where(rand() < half, 1 + (rand() < 0.5).long() + (rand() < 0.25).long(), torch.zeros_like(k))
    step = torch.cumsum(1 + gone - ins.long(), 0)
    src = up(start)[rid] + step - step[first[rid]]
    src = torch.minimum(src, up(toff[ctg + 1] - 1)[rid]).clamp_(min=0)
    b = tb[src]
    b = torch.where(ins | (up(rs.random(n) < 0.05)[rid]), _random_bases(tot, g, dev), b)
    code = ((b >> 1) ^ (b >> 2)) & 3
    other = _acgt((code + torch.randint(1, 4, (tot,), generator=g, device=dev, dtype=torch.uint8)) & 3)
    b = torch.where((rand() < up(sub)[rid].float()) & (b != 78), other, b)
    rev = up(rs.random(n) < 0.5)[rid]
    flipped = _complement(b[first[rid] + ln[rid] - 1 - k])
    return torch.where(rev, flipped, b), off


def _complement(b):
    t = torch.full((256,), 78, dtype=torch.uint8)
    t[list(_ACGT)] = torch.tensor(_ACGT[::-1], dtype=torch.uint8)
    return t.to(b.device)[b.long()]


def _inputs(c, seed):
    """Everything a case's calls are given: target and read sets (one per
    request of a served case) with their RAM loads, and the settings."""
    dev, g, rs = _tools(seed)
    tb, toff = _target(c, g, rs, dev)
    counts = [c["reads"]]
    if c["kind"] == "served":
        counts = rs.permutation(np.exp(np.linspace(0, math.log(c["reads"] + 0.5), c["requests"])).astype(np.int64))
    sets = [_reads(c, int(m), tb, toff, g, rs, dev) for m in counts]
    t_loads = api.ram_loads(np.diff(toff), max(T_RAM, c["t_vram"]))[1]
    q_loads = [api.ram_loads(np.diff(o), Q_RAM)[1] for _, o in sets]
    s = api.Setting(lmer=c["lmer"], stride=c["stride"], gap=c["gap"], local=c["local"], total_db=float(c["target_bp"]))
    return s, tb, toff, t_loads, sets, q_loads


def _placed(x, where):
    return x if where == "device" else x.cpu().pin_memory() if where == "pinned" else x.cpu().numpy()


_ENGINE = []


def _engine():
    """One context for the process, as a program keeps one."""
    if not _ENGINE:
        _ENGINE.append(api.Engine(0))
    return _ENGINE[0]


def prepare(case, seed):
    c, eng = case, _engine()
    s, tb, toff, t_loads, sets, q_loads = _inputs(c, seed)
    st = {"c": c, "eng": eng, "s": s, "toff": toff, "t_loads": t_loads, "q_loads": q_loads, "rest": {},
          "sets": [(_placed(b, c["where"]), o) for b, o in sets]}
    if torch.cuda.is_available():
        torch.cuda.synchronize()  # the library's streams read these buffers
    if c["kind"] == "window":
        t = api.joint_layout(tb.cpu().numpy(), toff, c["lmer"], 0, len(toff) - 1, False)
        st["ix"] = eng.hash_table_window(s, t[0], t[1], t[2], 0)
        b, o = st["sets"][0]
        st["window"] = api.joint_layout(b, o, c["lmer"], 0, len(o) - 1, True)
        return st
    st["tb"] = _placed(tb, c["where"])
    if c["kind"] != "job":
        st["T"] = eng.targets(s, st["tb"], toff, t_loads, c["t_vram"])
        del st["tb"]
    if c["kind"] == "served":
        st["server"] = api.Server(eng, st["T"], s, q_vram=Q_VRAM, q_ram=Q_RAM)
    if c["kind"] == "text":
        st["labels"] = (api.flat_labels(["r%d" % i for i in range(c["reads"])]),
                        api.flat_labels(["ctg%d" % i for i in range(len(toff) - 1)]))
    return st


#: Bytes of text per hit, and how many of them the first part of a text holds.
_LINE, _LINE_HEAD = 90, 55


def _two_parts(st, name, x, head, tail):
    """x as (its first `head` values, the others and zeros up to `tail`)."""
    n = len(x)
    if n > head + tail:
        raise RuntimeError("%s: %d values, more than the case allows" % (name, n))
    if name not in st["rest"]:
        st["rest"][name] = [np.zeros(tail, x.dtype), 0]
    rest, before = st["rest"][name]
    more = max(0, n - head)
    rest[:more] = x[head:]
    rest[more:before] = 0
    st["rest"][name][1] = more
    first = x[:head]
    if n < head:
        first = np.zeros(head, x.dtype)
        first[:n] = x
    return first, rest


def _outputs(st, r):
    """A result's hits in the two parts, and its offsets."""
    c = st["c"]
    out = {f: _two_parts(st, f, r[f], c["head"], c["tail"]) for f in r if f != "load_offsets"}
    if "load_offsets" in r:
        out["load_offsets"] = r["load_offsets"]
    return out


def run(st):
    c, eng, s = st["c"], st["eng"], st["s"]
    if c["kind"] == "window":
        return _outputs(st, eng.hit_list_window(s, st["ix"], *st["window"], 0))
    if c["kind"] == "served":
        srv = st["server"]
        ids = [srv.submit(b, o) for b, o in st["sets"]]
        got = [srv.poll(i) for i in ids]
        for i in ids:
            srv.release(i)
        return _outputs(st, {f: np.concatenate([r[f] for r in got]) for f in got[0]})
    b, o = st["sets"][0]
    if c["kind"] == "job":
        T = eng.targets(s, st["tb"], st["toff"], st["t_loads"], c["t_vram"])
        r = eng.map(s, T, b, o, st["q_loads"][0], Q_VRAM)
        T.close()
        return _outputs(st, r)
    r = eng.map(s, st["T"], b, o, st["q_loads"][0], Q_VRAM)
    if c["kind"] == "text":
        t = st["text"] = eng.format_tsv_text(st["T"], r, *st["labels"])
        text = np.frombuffer(t.view, np.uint8)
        return {"text": _two_parts(st, "text", text, _LINE_HEAD * c["head"], _LINE * c["tail"]),
                "evalue": _two_parts(st, "evalue", r["evalue"], c["head"], c["tail"])}
    return _outputs(st, r)


def work(case):
    """Bytes: target bases where the pass indexes them, read bases, 44 bytes per
    hit.  Operations: 13 per cell of the banded extension, one true hit per read
    and the expected hits of its repeat copies."""
    c = case
    lo, hi = c["len_lo"], c["len_hi"]
    mean = lo if lo == hi else (hi - lo) / math.log(hi / lo)
    reads = c["reads"]
    if c["kind"] == "served":
        reads = c["requests"] * max(1.0, c["reads"] / math.log(c["reads"] + 1))
    hits = reads * (0.95 + 0.3 * _copies(c))
    return {"bytes": float((c["target_bp"] if c["kind"] == "job" else 0) + reads * mean + 44.0 * hits),
            "flops": float(13 * hits * (2 * c["gap"] + 1) * max(0.0, mean - c["lmer"]))}


# ---------------------------------------------------------------- the same results in plain torch, 64-bit integers and doubles

_OPEN, _EXT, _MARGIN = -5, -2, -30000


def _code_of(b):
    """0..3 for A C G T, 4 for any other letter."""
    t = torch.full((256,), 4, dtype=torch.int64)
    t[list(_ACGT)] = torch.arange(4)
    return t.to(b.device)[b.long()]


def _kmers(code, at, l):
    """2-bit keys of the l letters from every position of `at`; -1 with a letter other than ACGT."""
    key = torch.zeros_like(at)
    bad = torch.zeros_like(at, dtype=torch.bool)
    pad = torch.cat([code, torch.full((l,), 4, dtype=code.dtype, device=code.device)])
    for i in range(l):
        x = pad[at + i]
        bad |= x > 3
        key = key * 4 + (x & 3)
    return torch.where(bad, -1, key)


def _windows(lens, budget):
    """Consecutive [begin, end) groups that grow while the next one's total stays below the budget."""
    out, b, n = [], 0, len(lens)
    cum = np.concatenate([[0], np.cumsum(lens)])
    while b < n:
        e = max(b + 1, min(n, int(np.searchsorted(cum, cum[b] + budget, side="left")) - 1))
        out.append((b, e))
        b = e
    return out


def _extend(code_t, t0, tlen, code_q, q0, rows, ti, step, gap, local):
    """One pass of the banded extension of many hits: (rows moved, end column, score, matches)."""
    W, dev = 2 * gap + 1, rows.device
    order = torch.argsort(rows, descending=True)
    t0, tlen, q0, rows_s, ti = t0[order], tlen[order], q0[order], rows[order], ti[order]
    n = len(rows)
    col = torch.arange(W, device=dev)
    init = torch.where(col < gap, _MARGIN, torch.where(col == gap, 0, (col - gap) * _EXT + _OPEN))
    S = init.repeat(n, 1)
    V = torch.where(col < gap, _MARGIN, init + _OPEN).repeat(n, 1)
    M = torch.where(col < gap, _MARGIN, 0).repeat(n, 1)
    bot = (gap + 1) * _EXT + _OPEN
    bs, bm = torch.zeros(n, dtype=torch.int64, device=dev), torch.zeros(n, dtype=torch.int64, device=dev)
    bc, be = torch.full((n,), -1, dtype=torch.int64, device=dev), torch.full((n,), gap, dtype=torch.int64, device=dev)
    left = rows_s.cpu().numpy()
    for r in range(int(left[0]) if n else 0):
        m = int(np.searchsorted(-left, -r, side="left"))  # the hits with more than r rows
        ib = ti[:m, None] + step * (r + col)
        out = (ib >= tlen[:m, None]) if step > 0 else (ib < 0)
        at = (t0[:m, None] + ib).clamp(0, len(code_t) - 1)
        inside = (t0[:m, None] + ib >= 0) & (t0[:m, None] + ib < len(code_t))
        tc = torch.where(out, 6, torch.where(inside, code_t[at], 4))
        eq = (tc == code_q[q0[:m] + step * r][:, None]) & (tc < 4)
        w = torch.where(tc == 6, -1000, torch.where(eq, 1, -3))
        wm = torch.where(tc == 6, -1000, eq.long())
        edge = torch.full((m, 1), bot, device=dev, dtype=torch.int64)
        nV = torch.maximum(torch.cat([S[:m, 1:], edge], 1) + _OPEN + _EXT,
                           torch.cat([V[:m, 1:], edge + _OPEN], 1) + _EXT)
        d = S[:m] + w
        P = torch.maximum(d, nV)
        Q = torch.where(nV >= d, torch.cat([M[:m, 1:], torch.zeros_like(edge)], 1), M[:m] + wm)
        # H along the row as a running maximum of P - 7 + 2c
        lead = torch.full((m, 1), _MARGIN + _EXT, device=dev, dtype=torch.int64)
        H = torch.cummax(torch.cat([lead, P[:, :-1] + _OPEN + _EXT - _EXT * (col[1:])], 1), 1)[0] + _EXT * col
        fromh = H >= P
        src = torch.cummax(torch.where(fromh, -1, col.expand(m, W)), 1)[0]
        S[:m], V[:m] = torch.maximum(P, H), nV
        M[:m] = torch.where(src < 0, _MARGIN, torch.gather(Q, 1, src.clamp(min=0)))
        if local:
            top, c = S[:m].max(1)
            c = (S[:m] == top[:, None]).long().argmax(1)
            up = top > bs[:m]
            bs[:m] = torch.where(up, top, bs[:m])
            bm[:m] = torch.where(up, torch.gather(M[:m], 1, c[:, None])[:, 0], bm[:m])
            bc[:m] = torch.where(up, r, bc[:m])
            be[:m] = torch.where(up, c, be[:m])
    if not local:
        bs = S.max(1)[0]
        be = (S == bs[:, None]).long().argmax(1)
        bm, low = torch.gather(M, 1, be[:, None])[:, 0], bs <= _MARGIN
        bs, bm, be = torch.where(low, _MARGIN, bs), torch.where(low, _MARGIN, bm), torch.where(low, -1, be)
        bc = rows_s - 1
    back = torch.empty_like(order)
    back[order] = torch.arange(n, device=dev)
    none = rows == 0
    return [torch.where(none, 0, x[back]) for x in (bc + 1, be - gap, bs, bm)]


def _window_hits(s, code_t, gw, lens, read_len, strand0, code_q, win_of_read):
    """(read, score, E-value) of one target window's hits, in result order."""
    dev, l, gap = code_t.device, s.lmer, s.gap
    ns = len(code_t) // s.stride
    keys = _kmers(code_t, torch.arange(ns, device=dev) * s.stride, l)
    keys, pos = torch.sort(keys, stable=True)
    slen = torch.repeat_interleave(read_len, 2)
    count = (slen - l + 1).clamp(min=0)
    strand = torch.repeat_interleave(torch.arange(len(slen), device=dev), count)
    qi = torch.arange(int(count.sum()), device=dev) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
    qk = _kmers(code_q, strand0[strand] + qi, l)
    a = torch.searchsorted(keys, qk)
    cnt = torch.searchsorted(keys, qk, right=True) - a
    cnt = torch.where((qk < 0) | ((s.cut_repeat != -1) & (cnt >= s.cut_repeat)), 0, cnt)
    strand, qi = torch.repeat_interleave(strand, cnt), torch.repeat_interleave(qi, cnt)
    e = torch.arange(int(cnt.sum()), device=dev) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt - a, cnt)
    p = pos[e] * s.stride
    tid = torch.searchsorted(gw, p, right=True) - 1
    ti = p - gw[tid]
    keep = ti + l <= lens[tid]
    if not s.local:
        keep &= (ti - qi + gap >= 0) & (ti - qi + slen[strand] - gap <= lens[tid])
    strand, qi, tid, ti = strand[keep], qi[keep], tid[keep], ti[keep]
    low = torch.argsort(((ti - qi + (1 << 20)) << 24) | qi, stable=True)
    o = low[torch.argsort((strand[low] << 24) | tid[low], stable=True)]
    v = [x[o] for x in (strand, qi, tid, ti)]
    for want_near in (True, False):  # isolated seeds go, then seeds near their predecessor
        strand, qi, tid, ti = v
        if not len(strand):
            return [torch.zeros(0, dtype=torch.int64, device=dev)] * 2 + [torch.zeros(0, dtype=torch.float64, device=dev)]
        near = (strand[1:] == strand[:-1]) & (tid[1:] == tid[:-1]) & ((ti[1:] - ti[:-1]).abs() <= s.width)
        near &= (ti - qi)[:-1] - (ti - qi)[1:] <= gap
        win = win_of_read[strand // 2]
        keep = torch.cat([torch.ones(1, dtype=torch.bool, device=dev), (near == want_near) | (win[1:] != win[:-1])])
        v = [x[keep] for x in v]
    strand, qi, tid, ti = v
    qlen = slen[strand]
    m1, e1, s1, _ = _extend(code_t, gw[tid], lens[tid], code_q, strand0[strand] + qi + l, qlen - qi - l, ti + l - gap, 1,
                            gap, s.local)
    m2, e2, s2, _ = _extend(code_t, gw[tid], lens[tid], code_q, strand0[strand] + qi - 1, qi, ti + gap - 1, -1, gap,
                            s.local)
    score = l + s1 + s2
    E = s.K * s.total_db * qlen.double() * torch.exp(-s.lambda_ * score.double())
    keep = l + m1 + m2 >= l + s.stride
    if s.cutoff != -1:
        keep &= E <= s.cutoff
    o_t, o_q = ti - m2 - e2, qi - m2
    cols = [x[keep] for x in (strand, qi, tid, ti, score, o_t, o_q)] + [E[keep]]
    strand, qi, tid, ti, score = cols[:5]
    o = torch.argsort(((strand & 1) << 60) | (tid << 32) | ti, stable=True)
    o = o[torch.argsort(((1 << 31) - score[o]) << 24 | ((1 << 23) - qi[o]), stable=True)]
    o = o[torch.argsort(strand[o] // 2, stable=True)]
    strand, qi, tid, ti, score, o_t, o_q, E = [x[o] for x in cols]
    same = (strand[1:] == strand[:-1]) & (tid[1:] == tid[:-1]) & (o_t[1:] == o_t[:-1]) & (o_q[1:] == o_q[:-1])
    keep = torch.cat([torch.ones(min(1, len(strand)), dtype=torch.bool, device=dev), ~same])
    return [strand[keep] // 2, score[keep], E[keep]]


def _exact_evalues(c, s, tb, toff, t_loads, rb, roff, q_loads):
    dev = tb.device
    lens = np.diff(roff)
    L = torch.from_numpy(lens).to(dev)
    off = torch.from_numpy(roff[:-1].copy()).to(dev)
    # both strands of every read, back to back
    rid = torch.repeat_interleave(torch.arange(len(lens), device=dev), L)
    k = torch.arange(int(roff[-1]), device=dev) - off[rid]
    both = torch.empty(2 * int(roff[-1]), dtype=torch.uint8, device=dev)
    both[2 * off[rid] + k] = rb
    both[2 * off[rid] + 2 * L[rid] - 1 - k] = _complement(rb)
    strand0 = torch.stack([2 * off, 2 * off + L], 1).reshape(-1)
    code_q = _code_of(both)
    win = np.zeros(len(lens), np.int64)
    if c["kind"] != "window":
        r0 = nw = 0
        for n in q_loads:
            for a, b in _windows(2 * (lens[r0:r0 + n] + c["lmer"] - 1), Q_VRAM):
                win[r0 + a:r0 + b] = nw
                nw += 1
            r0 += n
    win = torch.from_numpy(win).to(dev)
    parts, r0 = [], 0
    tl = np.diff(toff)
    for n in t_loads if c["kind"] != "window" else [len(tl)]:
        wins = _windows(tl[r0:r0 + n] + c["lmer"] - 1, c["t_vram"]) if c["kind"] != "window" else [(0, n)]
        for a, b in wins:
            seqs = [tb[toff[i]:toff[i + 1]] for i in range(r0 + a, r0 + b)]
            code_t = _code_of(torch.cat([x for q in seqs for x in (q, q[:c["lmer"] - 1])]))
            ln = tl[r0 + a:r0 + b]
            gw = np.concatenate([[0], np.cumsum(ln + c["lmer"] - 1)])[:-1]
            parts.append(_window_hits(s, code_t, torch.from_numpy(gw).to(dev), torch.from_numpy(ln).to(dev), L, strand0,
                                      code_q, win))
        r0 += n
    read, score, E = [torch.cat(x) for x in zip(*parts)]
    if len(parts) > 1:
        o = torch.argsort(score, descending=True, stable=True)
        E = E[o[torch.argsort(read[o], stable=True)]]
    return E.cpu().numpy()


def exact(case, seed):
    """The E-values of the pass (the path's only computed real numbers); whole numbers and text have no other value."""
    c = case
    s, tb, toff, t_loads, sets, q_loads = _inputs(c, seed)
    E = np.concatenate([_exact_evalues(c, s, tb, toff, t_loads, b, o, ql) for (b, o), ql in zip(sets, q_loads)])
    return {"evalue": _two_parts({"rest": {}}, "evalue", E, c["head"], c["tail"])}
