"""What the alignment stage is measured on: the calls a mapper makes, over the sizes they have.

Every case goes through the library's public entry points as a program that maps reads uses
them: the C ABI (include/sf_align.h) through its Python binding, with pinned host buffers for
pools, results and CIGARs, one device context for the process, plans and servers kept.

Paths
  call    one C-ABI call on one pair (`distance`, `affine_cigar`): latency
  plan    a device-resident batch: sf_plan_execute + sf_plan_download
  batch   a whole batch from host memory: sf_batch_run (descriptors and sequences in,
          results and CIGARs out)
  ends    span-end extensions of a hit batch over a transcript store: sf_extend_ends_batch
  sorted  the tie-break's sorted DP calls of a read batch: sf_sorted_batch
  serve   a burst of read batches through the serving loop: submit all, wait for all

Workloads (sizes of bench.py's configurations): reads of a fixed or log-normal length against
their own error-bearing copies (5-12% indel-heavy errors; 8% uniform errors for the plain edit
distances), each with `flank` unrelated bases on both sides where the text is a window.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from spearfish_gb300 import _abi
from spearfish_gb300 import batch as B
from spearfish_gb300 import serve as S
from spearfish_gb300 import tiebreak as T
from spearfish_gb300 import workloads as W
from spearfish_gb300.align import Affine, _aff

NOLIMIT = (1 << 64) - 1
SCORES = {"ont": Affine.ONT, "hifi": Affine.HIFI}
# Error profiles: (substitutions, insertions, deletions, indel weight inside homopolymers).
PROFILES = {"uniform": W.UNIFORM_211, "indel": W.ONT_INDEL, "hifi": W.HIFI}


def listed():
    return [
        # One read against one window: the mapper's single-pair distance call (latency).
        {"name": "one-distance", "path": "call", "what": "distance", "m": 1000, "mode": 0},
        # One read's banded alignment with its path: a single `affine` call (latency).
        {"name": "one-cigar", "path": "call", "what": "cigar", "m": 2000, "band": 128,
         "scores": "ont"},
        # Reads against flanked windows, Infix edit distance: the whole-read tie-break.
        {"name": "infix-1kb", "path": "plan", "what": "myers", "pairs": 10000, "len": 1000,
         "sigma": 0.0, "mode": 0, "cap": 0, "decoys": 0.0, "profile": "uniform", "rate": 0.08},
        # Capped Global distances, half of the candidates unrelated (rejected under the cap),
        # read lengths as sequenced.
        {"name": "capped-global", "path": "plan", "what": "myers", "pairs": 20000, "len": 900,
         "sigma": 0.6, "mode": 2, "cap": 220, "decoys": 0.5, "profile": "indel", "rate": 0.08},
        # Banded alignment with CIGARs, 2 kb reads, band 128.
        {"name": "cigar-2kb", "path": "plan", "what": "affine", "pairs": 20000, "len": 2000,
         "sigma": 0.0, "band": 128, "cigar": 1, "scores": "ont", "profile": "indel",
         "rate": 0.10},
        # The same pairs, scores only.
        {"name": "score-2kb", "path": "plan", "what": "affine", "pairs": 20000, "len": 2000,
         "sigma": 0.0, "band": 128, "cigar": 0, "scores": "ont", "profile": "indel",
         "rate": 0.10},
        # The uneven batch: 200 b - 20 kb reads, a distance and a banded CIGAR each, bands
        # 64-512 by length.
        {"name": "uneven", "path": "plan", "what": "both", "pairs": 25000, "len": 1200,
         "sigma": 0.8, "band": 0, "cigar": 1, "scores": "ont", "profile": "indel",
         "rate": 0.0},
        # A smaller uneven batch as one whole call from host memory.
        {"name": "uneven-call", "path": "batch", "what": "both", "pairs": 6000, "len": 1200,
         "sigma": 0.8, "band": 0, "cigar": 1, "scores": "ont", "profile": "indel",
         "rate": 0.0},
        # Read-end extension of whole 2 kb reads: X-drop, end bonus, clip cell, CIGAR.
        {"name": "window-2kb", "path": "plan", "what": "window", "pairs": 8000, "len": 2000,
         "sigma": 0.0, "band": 128, "cigar": 1, "scores": "ont", "profile": "indel",
         "rate": 0.10},
        # Span ends of a hit batch: both 20-200 base flanks of each hit, band 16, X-drop 50,
        # flanks sliced from the transcript store.
        {"name": "span-ends", "path": "ends", "hits": 40000, "flank": 200, "band": 16},
        # The tie-break's sorted calls: read ends and interior gaps against 1-9 isoform texts.
        {"name": "tie-break", "path": "sorted", "calls": 12000, "seg": 120, "band": 16},
        # The serving loop: a burst of read batches (1-320 reads), ONT cDNA and 10% HiFi reads.
        {"name": "served", "path": "serve", "requests": 10, "reads": 320},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["call", "plan", "plan", "plan", "batch", "batch", "ends", "sorted",
                       "serve"])
    if path == "call":
        what = rng.choice(["distance", "cigar"])
        c = {"path": path, "what": what, "m": _log(rng, 100, 8000)}
        if what == "distance":
            c["mode"] = rng.choice([0, 1, 2])
        else:
            c["band"] = _log(rng, 16, 256)
            c["scores"] = rng.choice(["ont", "hifi"])
        return c
    if path == "ends":
        return {"path": path, "hits": _log(rng, 64, 40000), "flank": _log(rng, 40, 400),
                "band": rng.choice([16, 24, 32])}
    if path == "sorted":
        return {"path": path, "calls": _log(rng, 64, 12000), "seg": _log(rng, 40, 300),
                "band": rng.choice([16, 24, 32])}
    if path == "serve":
        return {"path": path, "requests": rng.randint(2, 10), "reads": _log(rng, 8, 320)}
    what = rng.choice(["myers", "affine", "both", "window"])
    length = _log(rng, 300, 5000)
    c = {"path": path, "what": what, "len": length, "sigma": rng.choice([0.0, 0.3, 0.8])}
    # Pairs so that the batch's bases stay under those of the largest listed batch.
    c["pairs"] = _log(rng, 32, max(64, min(20000, 20_000_000 // length)))
    hifi = rng.random() < 0.25
    c["profile"] = "hifi" if hifi else "indel"
    c["rate"] = 0.01 if hifi else round(rng.uniform(0.05, 0.12), 3)
    if what == "myers":
        c["mode"] = rng.choice([0, 0, 1, 2])
        c["cap"] = rng.choice([0, 60, 250])
        c["decoys"] = rng.choice([0.0, 0.5])
    else:
        c["band"] = rng.choice([0, 64, 100, 128, 200, 256, 400])
        c["cigar"] = rng.choice([0, 1, 1])
        c["scores"] = "hifi" if hifi else "ont"
    return c


# ---- inputs ----------------------------------------------------------------------------------

_ctx = None


def context():
    """One device context for the process, as a mapper keeps one per device."""
    global _ctx
    if _ctx is None:
        _ctx = B.Context(0)
    return _ctx


def _pinned(n, dtype):
    """A pinned host array of n elements."""
    size = int(n) * np.dtype(dtype).itemsize
    t = torch.empty(max(16, size), dtype=torch.uint8, pin_memory=True)
    return t.numpy()[:size].view(dtype), t


def _lengths(case, gen):
    n = case["pairs"]
    if not case["sigma"]:
        return torch.full((n,), case["len"], dtype=torch.int64, device="cuda")
    z = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    x = torch.exp(math.log(case["len"]) + case["sigma"] * z).round()
    return x.clamp(200, 20000).to(torch.int64)


def _mutated(q, pair, rate, p, gen):
    """q's bases (of pairs `pair`) with errors at `rate` per pair: the read model of
    workloads.simulate, for all pairs at once.  Returns (bases, per-pair lengths)."""
    n, pairs = q.numel(), rate.numel()
    new = torch.ones(n, dtype=torch.bool, device="cuda")
    new[1:] = (q[1:] != q[:-1]) | (pair[1:] != pair[:-1])
    run = torch.cumsum(new, 0) - 1
    hp = torch.bincount(run)[run] >= 3
    share = hp.double().mean()
    bias = (1.0 / (1.0 - share + p.hp_bias * share)) * torch.where(hp, p.hp_bias, 1.0)
    r = rate[pair]
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    gone = u < r * p.dele * bias
    subs = ~gone & (u < r * p.dele * bias + r * p.sub)
    other = torch.randint(1, 4, (n,), generator=gen, device="cuda", dtype=torch.uint8)
    base = torch.where(subs, (q + other) & 3, q)
    ins = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) < r * p.ins * bias
    rand = torch.randint(0, 4, (n,), generator=gen, device="cuda", dtype=torch.uint8)
    ins_base = torch.where(hp, q, rand)
    two = torch.stack([base, ins_base], 1).reshape(-1)
    keep = torch.stack([~gone, ins], 1).reshape(-1)
    out = two[keep]
    lens = torch.bincount(pair.repeat_interleave(2)[keep], minlength=pairs)
    return out, lens


def _pairs(case, gen):
    """Reads and their texts: (pool on the device, read offsets, lengths, text offsets,
    lengths); the pool holds read 0, text 0, read 1, ..."""
    flank = 50 if case["what"] == "both" or (case["what"] == "myers" and case["mode"] == 0) else 0
    L = _lengths(case, gen)
    pairs = L.numel()
    pair = torch.repeat_interleave(torch.arange(pairs, device="cuda"), L)
    q = torch.randint(0, 4, (pair.numel(),), generator=gen, device="cuda", dtype=torch.uint8)
    rate = torch.full((pairs,), case["rate"], device="cuda", dtype=torch.float64)
    if not case["rate"]:
        rate = 0.05 + 0.07 * torch.rand(pairs, generator=gen, device="cuda", dtype=torch.float64)
    t, tl = _mutated(q, pair, rate, PROFILES[case["profile"]], gen)
    if case.get("decoys"):
        decoy = torch.rand(pairs, generator=gen, device="cuda") < case["decoys"]
        tpair = torch.repeat_interleave(torch.arange(pairs, device="cuda"), tl)
        rand = torch.randint(0, 4, (t.numel(),), generator=gen, device="cuda", dtype=torch.uint8)
        t = torch.where(decoy[tpair], rand, t)
    n = tl + 2 * flank
    step = L + n
    at = torch.cumsum(step, 0) - step
    pool = torch.randint(0, 4, (int(step.sum()),), generator=gen, device="cuda",
                         dtype=torch.uint8)

    def put(src, lens, where):
        start = torch.cumsum(lens, 0) - lens
        idx = torch.arange(src.numel(), device="cuda")
        pool[idx + torch.repeat_interleave(where - start, lens)] = src

    put(q, L, at)
    put(t, tl, at + L + flank)
    host = [x.cpu().numpy() for x in (at, L, at + L, n)]
    return pool, host, flank


def _jobs(case, gen):
    pool, (p_off, m, t_off, n), flank = _pairs(case, gen)
    pairs = m.size
    both = case["what"] == "both"
    jobs = B.new_jobs(pairs * (2 if both else 1))
    step = 2 if both else 1
    if case["what"] in ("myers", "both"):
        j = jobs[0::step]
        j["p_off"], j["m"], j["t_off"], j["n"] = p_off, m, t_off, n
        j["kind"], j["mode"] = B.JOB_MYERS, case.get("mode", 0)
        if case.get("cap"):
            j["k"] = case["cap"]
    if case["what"] != "myers":
        j = jobs[(1 if both else 0)::step]
        j["p_off"], j["m"], j["t_off"], j["n"] = p_off, m, t_off + flank, n - 2 * flank
        band = case["band"] or W.c3_band(m.astype(np.float64))
        j["band"], j["want_cigar"] = band, case["cigar"]
        if case["what"] == "window":
            j["kind"], j["mode"] = B.JOB_EXTEND_WINDOW, 1
            j["window"] = m + 20 + m // 10
            j["end_bonus"], j["xdrop"] = 5, 50
        else:
            j["kind"], j["mode"] = B.JOB_AFFINE, 2
    host, keep = _pinned(pool.numel(), np.uint8)
    keep[:pool.numel()].copy_(pool)
    return host, keep, jobs


def _buffers(jobs, ops_cap):
    """The caller's result and CIGAR buffers for one batch (zeroed: what no CIGAR fills stays
    zero)."""
    res, k0 = _pinned(len(jobs), B.RESULT_DTYPE)
    ops, k1 = _pinned(max(1, ops_cap), np.uint32)
    k0.zero_()
    k1.zero_()
    return res, ops, (k0, k1)


def _ops_cap(case):
    """Op slots for a batch's CIGARs: three a five bases of its expected length (10% errors
    make about one a nine), and room for a batch of few reads."""
    if not case.get("cigar"):
        return 1
    mean = max(200.0, case["len"]) * math.exp(case["sigma"] ** 2 / 2)
    return int(0.6 * mean * case["pairs"]) + 100_000


def _ptr(a, t):
    return a.ctypes.data_as(C.POINTER(t))


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    path = case["path"]
    if path == "call":
        c = {"what": "myers" if case["what"] == "distance" else "affine", "pairs": 1,
             "len": case["m"], "sigma": 0.0, "mode": case.get("mode", 2), "rate": 0.08,
             "profile": "indel"}
        pool, (p_off, m, t_off, n), _ = _pairs(c, gen)
        pool = pool.cpu().numpy()
        s.p = pool[p_off[0]:p_off[0] + m[0]].copy()
        s.t = pool[t_off[0]:t_off[0] + n[0]].copy()
        s.ops = np.zeros(3 * case["m"] + 64, np.uint32)
        s.sc = _aff(SCORES[case.get("scores", "ont")])
    elif path in ("plan", "batch"):
        s.pool, s.keep, s.jobs = _jobs(case, gen)
        s.res, s.ops, s.keep2 = _buffers(s.jobs, _ops_cap(case))
        s.sc = (SCORES[case.get("scores", "ont")],)
        if path == "plan":
            s.plan = B.Plan(context(), s.jobs, s.pool.size, s.sc)
            s.plan.upload(s.pool)
            s.plan.sync()
        else:
            s.scores = (_abi.Affine * 1)(_aff(s.sc[0]))
    elif path == "ends":
        _prepare_ends(s, case, np.random.default_rng(int(seed)))
    elif path == "sorted":
        _prepare_sorted(s, case, np.random.default_rng(int(seed)))
    else:
        _prepare_serve(s, case, np.random.default_rng(int(seed)))
    return s


def _edited(region, rng, rate=0.08):
    """Rows of `region` with substitutions at half of `rate` and one base dropped or doubled
    here and there at the other half, cut back to the row's width."""
    n, w = region.shape
    u = rng.random((n, w))
    move = np.where(u < rate / 4, 1, np.where(u < rate / 2, -1, 0))
    src = np.arange(w)[None, :] + np.cumsum(move, 1)
    out = np.take_along_axis(region, np.clip(src, 0, w - 1), 1)
    subs = (u >= rate / 2) & (u < rate)
    return np.where(subs, (out + rng.integers(1, 4, (n, w), dtype=np.uint8)) & 3, out)


def _prepare_ends(s, case, rng):
    """Hits over stored transcripts whose spans stop short of both read ends."""
    hits, most = case["hits"], case["flank"]
    n_tx, tx_len = 2000, 1600 + 4 * most
    tx = rng.integers(0, 4, (n_tx, tx_len), dtype=np.uint8)
    s.store = B.Store(context(), transcripts=list(tx))
    which = rng.integers(0, n_tx, hits)
    left = rng.integers(max(1, most // 10), most + 1, hits)
    right = rng.integers(max(1, most // 10), most + 1, hits)
    span = 300  # the anchored middle of the read
    start = rng.integers(most, tx_len - span - 2 * most, hits)  # the span's first tx base
    cols = np.arange(span + 2 * most)[None, :]
    region = tx[which[:, None], (start - most)[:, None] + cols]
    region[:, :most] = _edited(region[:, most - 1::-1][:, :most], rng)[:, ::-1]
    region[:, most + span:] = _edited(region[:, most + span:], rng)
    # Each read: its last `left` bases before the span, the span, `right` bases after it.
    keep = (cols >= (most - left)[:, None]) & (cols < (most + span + right)[:, None])
    lens = left + span + right
    s.pool, s.keep = _pinned(int(lens.sum()), np.uint8)
    s.pool[:] = region[keep]
    h = np.zeros(hits, dtype=T.HIT_DTYPE)
    h["read_off"] = np.cumsum(lens) - lens
    h["read_len"], h["tx_start"], h["tx_len"] = lens, s.store.starts[which], tx_len
    h["qstart"], h["qend"] = left, left + span
    h["tstart"], h["tend"] = start, start + span
    s.hits = h
    s.ends = {"sc": Affine.ONT, "band": case["band"], "end_bonus": 5, "xdrop": 50, "pad": 20,
              "pad_div": 10}


def _prepare_sorted(s, case, rng):
    """Read segments against the sorted distinct texts of 1-9 candidates: two read ends
    (extension cut at the shortest text) to one interior gap (Global)."""
    calls, spans, parts, at = [], [], [], 0
    n = case["calls"]
    segs = np.clip(np.round(np.exp(math.log(case["seg"]) + 0.5 * rng.standard_normal(n))), 12,
                   4 * case["seg"]).astype(np.int64)
    cs = (_abi.SortedCallT * n)()
    for i in range(n):
        m = int(segs[i])
        w = m + 20 + m // 10
        end = rng.random() < 0.67
        base = rng.integers(0, 4, w, dtype=np.uint8)
        read = base[:m].copy()
        hit = rng.random(m) < 0.06
        read[hit] = (read[hit] + 1) & 3
        drop = rng.random(m) < 0.03
        read = np.ascontiguousarray(read[~drop])
        texts = {}
        for _ in range(int(rng.integers(1, 10))):
            t = base[:w if end else m].copy()
            if t.size > 8 and rng.random() < 0.8:  # an isoform: a stretch replaced or skipped
                a = int(rng.integers(0, t.size - 4))
                b = int(rng.integers(a + 1, min(t.size, a + 40) + 1))
                if rng.random() < 0.5:
                    t[a:b] = rng.integers(0, 4, b - a, dtype=np.uint8)
                else:
                    t = np.concatenate([t[:a], t[b:]])
            texts[t.tobytes()] = t
        c = cs[i]
        c.p_off, c.m, c.first, c.band = at, read.size, len(spans), case["band"]
        parts.append(read)
        at += read.size
        ordered = [texts[k] for k in sorted(texts)]
        c.count = len(ordered)
        for t in ordered:
            spans.append((at, t.size))
            parts.append(t)
            at += t.size
        c.kind, c.mode, c.cut, c.xdrop = T.SORTED_AFFINE, 2, NOLIMIT, 2 ** 31 - 1
        if end:
            c.kind, c.mode = T.SORTED_EXTEND_CUT, 1
            c.window = max(w, max(t.size for t in ordered))
            c.end_bonus, c.xdrop, c.bonus_within_cut = 5, 50, 1
            c.cut = min(t.size for t in ordered)
    s.calls = cs
    s.spans = (_abi.SpanT * len(spans))(*[_abi.SpanT(o, k) for o, k in spans])
    s.pool, s.keep = _pinned(at, np.uint8)
    s.pool[:] = np.concatenate(parts)
    s.scores = (_abi.Affine * 1)(_aff(Affine.ONT))
    s.out = np.zeros(9 * n, dtype=np.dtype([("whole", "<i4"), ("cut", "<i4"),
                                                 ("cols", "<u8")]))


_server = None


def _prepare_serve(s, case, rng):
    global _server
    if _server is None:
        _server = S.Server(0, slots=8)
    s.requests = []
    for size in _batch_sizes(case):
        reads = [W.serving_read(rng, hifi=rng.random() < 0.1) for _ in range(size)]
        pool, jobs = W.serving_jobs(reads, B)
        host, keep = _pinned(pool.size, np.uint8)
        host[:] = pool
        s.requests.append((host, jobs, _buffers(jobs, 1000 * size + 20_000), keep))


def _batch_sizes(case):
    """Reads per request: log-uniform from 1 to the largest, the largest first."""
    n, most = case["requests"], case["reads"]
    return [max(1, round(most ** (1 - q / max(1, n - 1)))) for q in range(n)]


# ---- one pass ----------------------------------------------------------------------------------

def run(s):
    lib = _abi.load()
    path = s.case["path"]
    if path == "call":
        p, t = _ptr(s.p, C.c_uint8), _ptr(s.t, C.c_uint8)
        if s.case["what"] == "distance":
            d = C.c_uint32()
            _abi.check(lib.sf_distance(p, s.p.size, t, s.t.size, s.case["mode"], _abi.SF_NONE,
                                       C.byref(d)))
            return d.value
        out = _abi.CigarT()
        _abi.check(lib.sf_affine_cigar(p, s.p.size, t, s.t.size, 2, C.byref(s.sc),
                                       s.case["band"], _ptr(s.ops, C.c_uint32), s.ops.size,
                                       C.byref(out)))
        return [out.score, out.status, out.pattern_end, out.text_start, out.text_end,
                out.n_ops, s.ops.view(np.int32)]
    if path in ("plan", "batch"):
        used = C.c_uint64()
        if path == "plan":
            s.plan.execute()
            _abi.check(lib.sf_plan_download(s.plan.handle, _ptr(s.res, _abi.ResultT),
                                            _ptr(s.ops, C.c_uint32), s.ops.size,
                                            C.byref(used)))
        else:
            _abi.check(lib.sf_batch_run(context().handle, _ptr(s.pool, C.c_uint8), s.pool.size,
                                        _ptr(s.jobs, _abi.JobT), len(s.jobs), s.scores, 1,
                                        _ptr(s.res, _abi.ResultT), _ptr(s.ops, C.c_uint32),
                                        s.ops.size, C.byref(used)))
        return {"results": _fields(s.res), "ops": s.ops.view(np.int32), "used": used.value}
    if path == "ends":
        context().use_store(s.store)
        h = T.extend_ends_batch(context(), s.pool, s.ends, s.hits)
        return {k: h[k] for k in ("qstart", "qend", "tstart", "tend")}
    if path == "sorted":
        _abi.check(lib.sf_sorted_batch(context().handle, _ptr(s.pool, C.c_uint8), s.pool.size,
                                       s.scores, 1, s.calls, len(s.calls), s.spans,
                                       len(s.spans), _ptr(s.out, _abi.CutT)))
        return {k: s.out[k] for k in ("whole", "cut", "cols")}
    tickets = []
    for pool, jobs, _, _ in s.requests:
        t = C.c_uint64()
        _abi.check(lib.sf_server_submit(_server.handle, _ptr(pool, C.c_uint8), pool.size,
                                        _ptr(jobs, _abi.JobT), len(jobs), C.byref(t)))
        tickets.append(t)
    got = []
    for t, (_, _, (res, ops, _), _) in zip(tickets, s.requests):
        used, stats = C.c_uint64(), _abi.RequestStats()
        _abi.check(lib.sf_server_wait(_server.handle, t, 60_000, _ptr(res, _abi.ResultT),
                                      _ptr(ops, C.c_uint32), ops.size, C.byref(used),
                                      C.byref(stats)))
        got.append({"results": _fields(res), "ops": ops.view(np.int32), "used": used.value})
    return got


def _fields(res):
    """The result records as the words they are (views, no copy)."""
    return res.view(np.int32).reshape(len(res), -1)


# ---- what a pass cannot do without -------------------------------------------------------------

def _affine_work(rows, text, band, cigar):
    """(bytes, integer operations) of banded passes: sequences in, results and CIGARs out, and
    ten 32-bit operations a band cell, twelve where its traceback decisions are kept."""
    wide = np.minimum(2.0 * band + 1, text + 1.0)
    ops = float((rows * wide).sum()) * (12 if cigar else 10)
    out = 64.0 * len(rows) + (2.0 * float(rows.sum()) if cigar else 0.0)
    return float((rows + text).sum()) + out, ops


def work(case):
    path = case["path"]
    if path == "call":
        m = np.array([float(case["m"])])
        if case["what"] == "distance":
            return {"bytes": 2 * case["m"] + 4, "flops": 0.625 * case["m"] ** 2}
        b, f = _affine_work(m, m, case["band"], True)
        return {"bytes": b, "flops": f}
    if path in ("plan", "batch"):
        z = np.random.default_rng(1).standard_normal(case["pairs"])
        m = np.clip(np.exp(math.log(case["len"]) + case["sigma"] * z), 200, 20000) \
            if case["sigma"] else np.full(case["pairs"], float(case["len"]))
        b = f = 0.0
        if case["what"] in ("myers", "both"):
            b += float((2 * m).sum()) + 64.0 * m.size
            f += 0.625 * float((m * m).sum())
        if case["what"] != "myers":
            band = case["band"] or W.c3_band(m).astype(np.float64)
            x, y = _affine_work(m, m, band, case["cigar"])
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    if path == "ends":
        flank = np.full(2 * case["hits"], 0.55 * case["flank"])
        b, f = _affine_work(flank, 1.1 * flank + 20, case["band"], False)
        return {"bytes": b, "flops": f}
    if path == "sorted":
        seg = np.full(5 * case["calls"], 1.1 * case["seg"])
        b, f = _affine_work(seg, seg + 20, case["band"], False)
        return {"bytes": b, "flops": f}
    # A served read: its distance, its banded path and two 100-base extensions.
    m = np.full(sum(_batch_sizes(case)), 2100.0)
    x, y = _affine_work(m, m, 128.0, True)
    return {"bytes": x + float(m.sum()) * 2, "flops": y + 0.625 * float((m * m).sum()) * 1.8}


def exact(case, seed):
    """A single pair's result by the defining recurrence in 64-bit integers (the other cases'
    outputs are integers throughout, too many cells for plain numpy)."""
    if case["path"] != "call" or case["m"] > 2500:
        return None
    s = prepare(case, seed)
    p, t = s.p, s.t
    m, n = p.size, t.size
    if case["what"] == "distance":
        j = np.arange(n + 1, dtype=np.int64)
        row = np.zeros(n + 1, np.int64) if case["mode"] == 0 else j.copy()
        for i in range(1, m + 1):
            new = np.empty(n + 1, np.int64)
            new[0] = i
            new[1:] = np.minimum(row[1:] + 1, row[:-1] + (t != p[i - 1]))
            row = np.minimum.accumulate(new - j) + j
        return int(row[-1]) if case["mode"] == 2 else int(row.min())
    sc = SCORES[case["scores"]]
    below = case["band"] + max(0, m - n)
    above = case["band"] + max(0, n - m)
    low = np.int64(-(2 ** 40))
    j = np.arange(n + 1, dtype=np.int64)
    h = -(sc.open + sc.ext * j)
    h[0] = 0
    h[above + 1:] = low
    f = np.full(n + 1, low)
    for i in range(1, m + 1):
        f = np.maximum(h - sc.open, f) - sc.ext
        x = f.copy()
        x[1:] = np.maximum(x[1:], h[:-1] + np.where(t == p[i - 1], sc.mat, -sc.mis))
        out = (j < i - below) | (j > i + above)
        x[out] = f[out] = low
        e = np.full(n + 1, low)
        e[1:] = np.maximum.accumulate(x + sc.ext * j)[:-1] - sc.open - sc.ext * j[1:]
        h = np.maximum(x, e)
        h[out] = low
    return [int(h[n]), 0, m, 0, n, None, None]
