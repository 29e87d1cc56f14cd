"""The anti-diagonal 16-bit kernel (sf_wave16_impl.cuh) against the oracle: scores, end cells,
DP cells and CIGARs of Global and Prefix banded passes, bit-exact, where its layout can go wrong
-- every class filled to its last band cell, several passes of uneven length to a warp, bands
that start at column 0 for many rows, one-base sequences, row steps around the stores (4), the
window chunks (16) and the rebase (32), paths along the band's edges, long passes, score sets on
both sides of its admission rule; for Prefix passes the clip cell, the X-drop stop at any row, the
last row's best column and texts that end inside the band."""
import json

import numpy as np
import pytest

import oracle as O
import refcases as R

pytestmark = pytest.mark.gpu

# Few passes run one to a warp (or a team), as do those that take long against the whole batch;
# batches of more passes than this, with enough other work (`_ballast`), several to a warp.
PACKED = 3400


def _ballast():
    """The same wide score-only pass many times: a few milliseconds of device time."""
    rng = np.random.default_rng(26)
    q = rng.integers(0, 4, 3000).tolist()
    return [(q, R.mutate(q, R.rand_edits(rng, 200, 3000)), 600, 0, 0)] * 2400


@pytest.fixture(scope="module")
def ctx():
    from spearfish_gb300 import build
    build.build()
    from spearfish_gb300 import batch as B
    c = B.Context(0)
    yield c
    c.close()


def _run(ctx, rows, scores):
    """rows: (pattern, text, band, cigar, score index).  Returns the output and the plan's
    (kind, cells a lane, lanes) buckets."""
    from spearfish_gb300 import batch as B
    pb = B.PoolBuilder()
    jobs = B.new_jobs(len(rows))
    for j, (p, t, band, cig, sci) in zip(jobs, rows):
        j["p_off"], j["m"] = pb.add(p), len(p)
        j["t_off"], j["n"] = pb.add(t), len(t)
        j["kind"], j["mode"], j["band"], j["want_cigar"] = B.JOB_AFFINE, 2, band, cig
        j["sc_index"] = sci
    plan = B.Plan(ctx, jobs, pb.size, scores)
    try:
        plan.upload(pb.build())
        plan.execute()
        out = plan.download()
        plan.execute()  # replayed from the plan's graph
        again = plan.download()
        kinds = {(b["kind"], b["c"], b["lanes"]) for b in json.loads(plan.describe())["buckets"]}
    finally:
        plan.close()
    assert np.array_equal(out.results, again.results) and np.array_equal(out.ops, again.ops)
    return out, kinds


def _check(rows, out, scores):
    for q, (p, t, band, cig, sci) in enumerate(rows):
        r = out.results[q]
        o = O.traceback(p, t, O.TB_AFFINE, O.GLOBAL, scores[sci], band)
        where = (q, len(p), len(t), band, sci)
        assert (int(r["status"]), int(r["score"]), int(r["text_end"]), int(r["pattern_end"])) == \
            (0, o["score"], len(t), len(p)), where
        if cig:
            assert out.cigar(q) == o["cigar"], where


def _noisy(rng, m, rate):
    q = rng.integers(0, 4, m)
    return q.tolist(), R.mutate(q.tolist(), R.rand_edits(rng, int(m * rate), m))


def _shifted(rng, m, d):
    """A pair whose path leaves the main diagonal by d columns and comes back."""
    q = rng.integers(0, 4, m).tolist()
    cut = m // 2
    if d > 0:
        t = q[:cut] + rng.integers(0, 4, d).tolist() + q[cut:m - d]
    else:
        t = q[:cut] + q[cut - d:] + rng.integers(0, 4, -d).tolist()
    return q, t


@pytest.mark.parametrize("packed", [False, True])
def test_every_class_to_its_last_cell(ctx, packed):
    """Bands whose cells fill each class exactly, miss it by one, or pass it by one; paths that
    touch both band edges."""
    rng = np.random.default_rng(2601 + packed)
    rows = []
    caps = (48, 64, 72, 80, 96, 120, 128, 144, 160, 192, 200, 240, 256, 288, 320, 384, 400, 480,
            512, 640, 768, 1024, 1280, 1536)
    for cap in caps:
        for w in (cap - 1, cap, cap + 1):
            band, extra = (w - 2) // 2, (w - 2) % 2
            m = band + 30 + int(rng.integers(0, 90))
            d = int(rng.integers(-band, band + 1))
            p, t = _shifted(rng, m, d)
            t = (t + rng.integers(0, 4, extra).tolist())
            rows.append((p, t, band, 1 + 0 * cap, int(rng.integers(0, 2))))
    while packed and len(rows) < PACKED:
        band = int(rng.integers(1, 70))
        p, t = _noisy(rng, int(rng.integers(band + 2, 4 * band + 40)), 0.1)
        rows.append((p, t, band, int(rng.integers(0, 2)), int(rng.integers(0, 2))))
    scores = (R.ONT, R.HIFI)
    out, kinds = _run(ctx, rows + (_ballast() if packed else []), scores)
    assert len(set(out.results["score"][len(rows):].tolist())) <= 1
    wave = {(c, n) for k, c, n in kinds if k == "wave16"}
    want = {(16, 3), (24, 4), (40, 8), (48, 10), (32, 16), (48, 32)} if packed else \
        {(16, 8), (16, 16), (16, 32), (16, 62), (16, 92), (16, 122)}
    assert wave >= want, sorted(kinds)
    _check(rows, out, scores)


@pytest.mark.parametrize("packed", [False, True])
def test_small_and_uneven(ctx, packed):
    """One to a few dozen bases, every remainder of the row steps, passes of very different
    length side by side, bands wider than half the sequences."""
    rng = np.random.default_rng(2611 + packed)
    rows = []
    for m in list(range(1, 70)) + [127, 128, 129]:
        p, t = _noisy(rng, m, 0.15)
        t = t or [int(rng.integers(0, 4))]
        rows.append((p, t, int(rng.integers(0, max(1, m // 2) + 1)), m % 3 != 0, m % 2))
    rows.append(([0], [3], 0, 1, 0))
    rows.append(([0, 1, 2, 3] * 10, [2] * 75, 3, 1, 0))
    for _ in range(PACKED - len(rows) if packed else 40):
        m = int(np.exp(rng.uniform(np.log(4), np.log(600))))
        rate = float(rng.choice([0.0, 0.05, 0.3]))
        p, t = _noisy(rng, m, rate)
        if rng.random() < 0.15:
            t = rng.integers(0, 2, int(rng.integers(1, 2 * m + 2))).tolist()  # unrelated
        rows.append((p, t or [1], int(rng.integers(0, min(60, m) + 1)), int(rng.integers(0, 2)),
                     int(rng.integers(0, 2))))
    scores = (R.ONT, R.HIFI)
    out, _ = _run(ctx, rows + (_ballast() if packed else []), scores)
    _check(rows, out, scores)


def test_long_passes(ctx):
    """Thousands of row steps: identical sequences (the largest field climbs most), unrelated
    ones (it hardly moves), 10% errors; widths of the widest classes."""
    rng = np.random.default_rng(2621)
    rows = []
    for m, band, kind in ((20000, 40, "same"), (9000, 64, "unrelated"), (12000, 512, "noisy"),
                          (4000, 700, "noisy"), (3000, 700, "same"), (2500, 620, "unrelated")):
        q = rng.integers(0, 4, m).tolist()
        t = list(q) if kind == "same" else rng.integers(0, 4, m).tolist() \
            if kind == "unrelated" else R.mutate(q, R.rand_edits(rng, m // 10, m))
        rows += [(q, t, band, cig, sci) for cig in (0, 1) for sci in (0, 1)]
    scores = (R.ONT, R.HIFI)
    out, kinds = _run(ctx, rows, scores)
    assert any(k == "wave16" for k, _, _ in kinds), kinds
    _check(rows, out, scores)


def test_admission(ctx):
    """Score sets the kernel takes (mis = 2 ext, open >= 1) at its bounds, and ones it leaves to
    the row kernels: the same results either way."""
    rng = np.random.default_rng(2631)
    scores = ((3, 2, 1, 1), (7, 0, 5, 0), (0, 4, 1, 2), (59, 2, 900, 1), (61, 2, 5, 1),
              (20, 20, 10, 10), (2, 4, 0, 2), (2, 5, 4, 2), (2, 3, 4, 2), (0, 0, 1, 0))
    rows = []
    for sci in range(len(scores)):
        for band in (0, 5, 60, 150, 230, 330):
            p, t = _noisy(rng, int(rng.integers(max(20, band), 900)), 0.15)
            rows.append((p, t, band, 1, sci))
            p, t = _shifted(rng, 2 * band + 50, int(rng.integers(-band, band + 1)))
            rows.append((p, t, band, 1, sci))
    out, kinds = _run(ctx, rows, scores)
    assert {"wave16", "affine16"} <= {k for k, _, _ in kinds}, kinds
    _check(rows, out, scores)


def _run_prefix(ctx, rows, scores, rows_only=False):
    """rows: (pattern, text, band, window or None, xdrop, end bonus, cigar, score index); window
    None: an affine pass in Prefix mode, else an extension."""
    import os
    from spearfish_gb300 import batch as B
    pb = B.PoolBuilder()
    jobs = B.new_jobs(len(rows))
    for j, (p, t, band, win, xd, bonus, cig, sci) in zip(jobs, rows):
        j["p_off"], j["m"] = pb.add(p), len(p)
        j["t_off"], j["n"] = pb.add(t), len(t)
        j["band"], j["want_cigar"], j["sc_index"], j["mode"] = band, cig, sci, R.PREFIX
        j["kind"] = B.JOB_AFFINE if win is None else B.JOB_EXTEND_WINDOW
        if win is not None:
            j["window"], j["xdrop"], j["end_bonus"] = win, xd, bonus
    old = os.environ.get("SF_AFFINE16_LANES")
    if rows_only:
        os.environ["SF_AFFINE16_LANES"] = "32"
    try:
        plan = B.Plan(ctx, jobs, pb.size, scores)
        try:
            plan.upload(pb.build())
            plan.execute()
            out = plan.download()
            kinds = {(b["kind"], b["c"], b["lanes"]) for b in json.loads(plan.describe())["buckets"]}
        finally:
            plan.close()
    finally:
        if rows_only:
            if old is None:
                del os.environ["SF_AFFINE16_LANES"]
            else:
                os.environ["SF_AFFINE16_LANES"] = old
    return out, kinds


def _check_prefix(rows, out, scores):
    for q, (p, t, band, win, xd, bonus, cig, sci) in enumerate(rows):
        r, sc = out.results[q], scores[sci]
        where = (q, len(p), len(t), band, win, xd, sci)
        got = (int(r["status"]), int(r["score"]), int(r["pattern_end"]), int(r["text_end"]))
        if win is None:
            o = O.traceback(p, t, O.TB_AFFINE, O.PREFIX, sc, band)
            assert got == (0, o["score"], len(p), o["end_j"]), where
        else:
            o = O.traceback(p, t, O.TB_EXTEND, O.PREFIX, sc, band, win, bonus, xd)
            assert got == (0, o["score"], o["end_i"], o["end_j"]), where
            assert (*got[1:], int(r["text_read"])) == \
                O.affine_extend_window(p, t, win, sc, band, bonus, xd), where
        if cig:
            assert out.cigar(q) == o["cigar"], where


@pytest.mark.parametrize("packed", [False, True])
def test_prefix(ctx, packed):
    rng = np.random.default_rng(2641 + packed)
    rows = []

    def add(p, t, band, extend=True):
        t = t or [int(rng.integers(0, 4))]
        win = len(t) + int(rng.integers(0, 40)) if extend else None
        xd = int(rng.choice([0, 3, 8, 20, 50, R.I32_MAX]))
        rows.append((p, t, band, win, xd, int(rng.integers(0, 9)), int(rng.integers(0, 2)),
                     int(rng.integers(0, 2))))

    # Bands that fill each class, miss it by one or pass it by one, rows that end past, at and
    # before the text's end.
    for cap in (48, 64, 72, 80, 96, 128, 160, 192, 256, 320, 512, 768, 1024):
        for w in (cap - 1, cap, cap + 1):
            band, extra = (w - 2) // 2, (w - 2) % 2
            for cut in (0, 7, 40):
                m = band // 2 + 30 + int(rng.integers(0, 90))
                p, t = _shifted(rng, m, int(rng.integers(-(m // 3), m // 3 + 1)))
                t = t[:max(1, m - cut)] + rng.integers(0, 4, extra).tolist()
                # The window's geometry is the text's: below + above + 1 = w.
                rows.append((p[:len(t) - extra] if cut else p, t, band, len(t), 50, 5, 1, cap % 3 % 2))
                add(p, t, band, extend=False)
        if cap >= 512:
            # (Short patterns in wide bands run on the row kernel.)
            for w in (cap - 1, cap):
                p, t = _shifted(rng, 2 * cap, cap // 3)
                rows.append((p, t + rng.integers(0, 4, w % 2).tolist(), (w - 2) // 2, None,
                             R.I32_MAX, 0, 1, w % 2))
    for m in list(range(1, 60)) + [127, 128, 129, 400]:
        p, t = _noisy(rng, m, 0.15)
        add(p, t + rng.integers(0, 4, int(rng.integers(0, 30))).tolist(), int(rng.integers(0, 20)))
        add(p, t[:max(1, len(t) - int(rng.integers(0, 10)))], int(rng.integers(0, 20)), extend=False)
    # Extensions that go wrong part of the way: the X-drop stops at any row.
    for _ in range(PACKED - len(rows) if packed else 200):
        m = int(np.exp(rng.uniform(np.log(8), np.log(500))))
        good = int(rng.integers(0, m + 1))
        p, t = _noisy(rng, m, float(rng.choice([0.0, 0.05, 0.12])))
        t = t[:good] + rng.integers(0, 4, max(0, m + 20 - good)).tolist()
        add(p, t, int(rng.integers(1, 40)), extend=rng.random() < 0.8)
    scores = (R.ONT, R.HIFI)
    checked = len(rows)
    if packed:
        rows += [(p, t, b, None, R.I32_MAX, 0, 0, sci) for p, t, b, _, sci in _ballast()]
    out, kinds = _run_prefix(ctx, rows, scores)
    wave = {(c, n) for k, c, n in kinds if k == "wave16x"}
    want = {(16, 3), (24, 4), (32, 4), (32, 10), (32, 32)} if packed else \
        {(16, 8), (16, 16), (16, 32), (16, 62), (32, 32)}
    assert wave >= want, sorted(kinds)
    _check_prefix(rows[:checked], out, scores)
    # The row kernels give the same.
    ref, rkinds = _run_prefix(ctx, rows, scores, rows_only=True)
    assert not any(k.startswith("wave") for k, _, _ in rkinds)
    for f in ("score", "pattern_end", "text_start", "text_end", "text_read", "cells", "n_ops",
              "status"):
        assert np.array_equal(out.results[f], ref.results[f]), f
    assert np.array_equal(out.ops, ref.ops)


def test_prefix_long(ctx):
    """Thousands of row steps with every row's maximum in order, up to the widest class."""
    rng = np.random.default_rng(2651)
    rows = []
    for m, band in ((9000, 16), (6000, 128), (4000, 300), (3000, 480)):
        for kind in ("noisy", "half"):
            q = rng.integers(0, 4, m).tolist()
            t = R.mutate(q, R.rand_edits(rng, m // 10, m))
            if kind == "half":
                t = t[:m // 2] + rng.integers(0, 4, m // 2).tolist()
            for xd in (50, 400, R.I32_MAX):
                rows.append((q, t, band, len(t) + 60, xd, 5, 1, int(rng.integers(0, 2))))
    scores = (R.ONT, R.HIFI)
    out, kinds = _run_prefix(ctx, rows, scores)
    assert ("wave16x", 16, 32) in kinds and ("wave16x", 16, 92) in kinds, kinds
    _check_prefix(rows, out, scores)


@pytest.mark.parametrize("packed", [False, True])
def test_wide_bands(ctx, packed):
    """Bands past one warp's cells: Global and Prefix classes of teams filled to their last cell,
    missed or passed by one; paths along either edge (the largest spread of a row), X-drop stops
    in every part, score sets on both sides of what the widest classes take."""
    rng = np.random.default_rng(2661 + packed)
    scores = (R.ONT, R.HIFI, (1, 6, 4, 3), (3, 2, 900, 1), (5, 4, 4, 2), (0, 2, 1, 1))
    rows = []
    for cap in (992, 1024, 1472, 1952, 1984, 2432, 2912, 2944, 3392):
        for w in (cap - 1, cap, cap + 1):
            for edge in (0, 1):
                band = int(rng.integers(1, 90)) if edge else (w - 2) // 2
                extra = w - 2 * band - 2 + (w % 2)  # below + above + 1 = w, `below` odd or even
                m = max(band // 2 + 40, w // 4 + 20) + int(rng.integers(0, 60))
                q = rng.integers(0, 4, m).tolist()
                fill = rng.integers(0, 4, max(0, extra + band)).tolist()
                good = R.mutate(q, R.rand_edits(rng, int(m * rng.choice([0.0, 0.1])), m))
                t = (fill + good if edge and rng.random() < 0.5 else good + fill)[:m + extra]
                t += rng.integers(0, 4, m + extra - len(t)).tolist()
                xd = int(rng.choice([8, 50, 2000, R.I32_MAX]))
                rows.append((q, t, band, len(t), xd, 5, 1, len(rows) % len(scores)))
                rows.append((q, t, band, None, R.I32_MAX, 0, int(edge), (len(rows) // 2) % 3))
        q, t = _noisy(rng, 2 * cap, 0.1)
        for xd in (50, R.I32_MAX):
            rows.append((q, t + rng.integers(0, 4, cap - 200 - len(t) + 2 * cap).tolist(), 98,
                         3 * cap - 200, xd, 5, 1, len(rows) % 2))
    checked = len(rows)
    if packed:
        rows += [(p, t, b, None, R.I32_MAX, 0, 0, sci) for p, t, b, _, sci in _ballast() * 2]
    out, kinds = _run_prefix(ctx, rows, scores)
    wave = {(c, n) for k, c, n in kinds if k == "wave16x"}
    want = {(32, 62), (32, 92), (32, 122)} if packed else \
        {(16, 62), (16, 92), (16, 122), (16, 152), (16, 182), (16, 212)}
    assert wave >= want, sorted(kinds)
    _check_prefix(rows[:checked], out, scores)

    grows = []
    for w in (1536, 1537, 1952, 1953, 2432, 2912, 3392, 3393):
        band, extra = (w - 2) // 2, (w - 2) % 2
        for d in (-band, 0, band):
            p, t = _shifted(rng, band + 30 + int(rng.integers(0, 90)), d)
            grows.append((p, t + rng.integers(0, 4, extra).tolist(), band, 1, len(grows) % 2))
    gout, gkinds = _run(ctx, grows + (_ballast() if packed else []), scores)
    assert {(16, 152), (16, 182), (16, 212)} <= {(c, n) for k, c, n in gkinds if k == "wave16"}
    _check(grows, gout, scores)


@pytest.mark.parametrize("calls", [120, 3600])
def test_prefix_cut(ctx, calls):
    """Sorted-texts extensions with a cut column: left of the band, in it at any parity, at and
    past the text's end; X-drop stops in every part, even and odd last cells, bands of each class
    (a few calls run one pass a warp, many several)."""
    from spearfish_gb300 import tiebreak as T
    rng = np.random.default_rng(2671)
    scores = (R.ONT, R.HIFI)
    got_calls, want = [], []
    for q in range(calls):
        m = int(np.exp(rng.uniform(np.log(1), np.log(120 if q % 40 else 1500))))
        band = int(rng.choice([0, 1, 5, 16, 24, 32, 47])) if q % 40 else int(rng.integers(60, 400))
        base = rng.integers(0, 4, m + int(rng.integers(0, 40))).tolist()
        p = R.mutate(base[:m], R.rand_edits(rng, m // 12, m)) or [1]
        texts = sorted({tuple(R.mutate(base, R.rand_edits(rng, int(rng.integers(0, 6)), len(base))))
                        or (0,) for _ in range(int(rng.integers(1, 5)))})
        texts = [list(t) for t in texts]
        n = min(len(t) for t in texts)
        cut = int(rng.choice([0, 1, max(0, n - 3), n, n + 50, int(rng.integers(0, n + 1))]))
        xd = int(rng.choice([0, 6, 20, 50, R.I32_MAX]))
        bonus, track, within = int(rng.integers(0, 8)), bool(q & 1), bool(q & 2)
        diag, w, sci = bool(rng.random() < 0.2), max(len(t) for t in texts) + int(rng.integers(0, 30)), q % 2
        got_calls.append(dict(kind=T.SORTED_EXTEND_CUT, read=p, texts=texts, band=band,
                              end_bonus=bonus, xdrop=xd, diagonal=diag, window=w, cut=cut,
                              track_cut=track, bonus_within_cut=within, sc_index=sci))
        want.append(O.affine_extend_sorted_cut_bonus(p, texts, scores[sci], band, bonus, xd, diag,
                                                     w, cut, track, within))
    got = T.sorted_batch(ctx, got_calls, scores=scores)
    for q in range(calls):
        assert got[q] == want[q], (q, got_calls[q])


@pytest.mark.parametrize("op", [255, 256, 257, 300, 900])
def test_wide_prefix_open(ctx, op):
    """Large gap-open costs on both sides of what the classes past 1,024 cells take (a cell no
    path reaches gives up the opening too), at their first and last widths and below them."""
    rng = np.random.default_rng(2681 + op)
    scores = ((3, 2, op, 1), (3, 0, op, 0), (0, 2, op, 1))
    for cells in (1024, 1025, 1222, 1984, 3392, 1026):
        rows = []
        half = (cells - 2) // 2
        wide = (half | 1) + half + (cells - 2) % 2 + 1 > 1024
        for sci in range(len(scores)):
            for kind in ("noisy", "shifted", "half"):
                band, extra = (cells - 2) // 2, (cells - 2) % 2
                m = cells // 2 + 300 + int(rng.integers(0, 60))
                p, t = _noisy(rng, m, 0.05) if kind == "noisy" else \
                    _shifted(rng, m, int(rng.integers(-m // 3, m // 3 + 1)))
                if kind == "half":
                    t = t[:m // 2] + rng.integers(0, 4, m).tolist()
                t = (t + rng.integers(0, 4, m).tolist())[:m + extra]
                rows.append((p, t, band, None, R.I32_MAX, 0, 1, sci))
                rows += [(p, t, band, len(t), xd, 5, 1, sci) for xd in (50, R.I32_MAX)]
        out, kinds = _run_prefix(ctx, rows, scores)
        team = any(k == "wave16x" and lanes > 32 for k, _, lanes in kinds)
        assert any(k == "wave16x" for k, _, _ in kinds) == (op <= 256 or not wide), (cells, kinds)
        assert team == (op <= 256 and wide), (cells, kinds)
        _check_prefix(rows, out, scores)
