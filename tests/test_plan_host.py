"""The plan build's host phases on the CPU (tests/plan_check.cu): which kernel class each job gets
and the sizes the plan takes."""
import json
import os
import subprocess

import numpy as np
import pytest

import refcases as R

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from spearfish_gb300 import build
    lib = build.build()
    exe = str(tmp_path_factory.mktemp("plan") / "plan_check")
    cmd = [build.nvcc(), *build.ARCH, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I", build.INCLUDE,
           os.path.join(ROOT, "tests", "plan_check.cu"), lib, "-o", exe,
           "-Xlinker", "-rpath," + os.path.dirname(lib)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(jobs, scores=(R.ONT,), pool_bytes=None, sms=152, shared=False):
        if pool_bytes is None:
            pool_bytes = int(max((jobs["p_off"] + jobs["m"]).max(), (jobs["t_off"] + jobs["n"]).max()))
        path = exe + ".in"
        with open(path, "wb") as f:
            np.array([sms, pool_bytes, len(scores), len(jobs)], np.uint64).tofile(f)
            np.array([tuple(s) for s in scores], np.int32).tofile(f)
            jobs.tofile(f)
        out = subprocess.run([exe, path] + ["shared"] * shared, capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, out.stdout + out.stderr
        plan = json.loads(out.stdout)
        plan["kinds"] = [plan["plan"]["buckets"][b]["kind"] for b in plan["job_buckets"]]
        return plan
    return run


def _jobs(rows):
    """rows: dicts of job fields; patterns and texts one after another in the pool."""
    from spearfish_gb300 import batch as B
    jobs, at = B.new_jobs(len(rows)), 0
    for j, r in zip(jobs, rows):
        j["p_off"], j["t_off"] = at, at + r["m"]
        at += r["m"] + r["n"]
        for k, v in r.items():
            j[k] = v
    return jobs


@pytest.mark.parametrize("ext", [0, 1])
def test_wide_prefix_open(check, ext):
    """A cell no path reaches gives up a gap's opening: four times it at most what such cells hold,
    256 in the classes past 1,024 cells, and past 900 in no class."""
    from spearfish_gb300 import batch as B
    rows, want, scores = [], [], []
    for op in (255, 256, 257, 300, 900, 901):
        scores.append((3, 2 * ext, op, ext))
        for cells in (1023, 1025, 1222, 1984, 3391):
            for kind in (B.JOB_AFFINE, B.JOB_EXTEND_WINDOW):
                rows.append(dict(m=2000, n=2000, band=(cells - 1) // 2, kind=kind, mode=R.PREFIX,
                                 window=2000, xdrop=50, sc_index=len(scores) - 1, want_cigar=1))
                # below + above + 1 cells, below made odd.
                below = (cells - 1) // 2
                w = (below | 1) + below + 1
                want.append(op <= (256 if w > 1024 else 900))
    plan = check(_jobs(rows), scores)
    for r, k, ok in zip(rows, plan["kinds"], want):
        assert (k == "wave16x") == ok, (r, scores[r["sc_index"]], k)


@pytest.mark.parametrize("count", [1, 40, 4000])
@pytest.mark.parametrize("m,n,band", [(1000, 1060, 600), (1000, 650, 600), (400, 460, 300), (90, 100, 30),
                                      (60, 300, 120), (2000, 2100, 64)])
def test_estimate_is_an_upper_bound(check, m, n, band, count):
    """plan_bytes_estimate, which the server admits requests by, against what the plan takes: short
    patterns in wide bands, whose passes run on rows or on a team by how many there are."""
    from spearfish_gb300 import batch as B
    for kind in (B.JOB_AFFINE, B.JOB_EXTEND_WINDOW):
        for cigar in (0, 1):
            row = dict(m=m, n=n, band=band, kind=kind, mode=R.PREFIX, window=n, xdrop=100, want_cigar=cigar)
            plan = check(_jobs([row] * count))
            assert plan["estimate"] >= plan["needs"], (plan["kinds"][0], plan["estimate"], plan["needs"])


@pytest.mark.parametrize("others,pairs", [(700, 300), (100, 40), (20, 1500), (3000, 900)])
def test_trial_plans_keep_the_classes(check, others, pairs):
    """The autotuner times the passes of one class in a plan of their own, which is smaller: they
    must get the same default class there, or the candidates it names would not be what runs."""
    from spearfish_gb300 import batch as B
    rows = [dict(m=500 + 7 * (q % 50), n=560, band=40, kind=B.JOB_AFFINE, mode=R.GLOBAL, want_cigar=1)
            for q in range(others)]
    rows += [dict(m=m, n=m, kind=B.JOB_MYERS, mode=R.INFIX) for m in (700, 40 * 64, 100 * 64, 200 * 64)
             for _ in range(pairs // 4)]
    assert check(_jobs(rows))["strays"] == 0


@pytest.mark.parametrize("count", [1, 12, 2047, 50000])
@pytest.mark.parametrize("text", [300, 4096, 40000, 70000])
def test_shared_sequences(check, text, count):
    """Many reads that name a few transcripts in turn: each transcript is packed once where its
    copies would weigh, and every pass finds its own sequences."""
    from spearfish_gb300 import batch as B
    rng = np.random.default_rng(31)
    texts = 7
    jobs = B.new_jobs(count)
    jobs["kind"], jobs["mode"] = B.JOB_MYERS, R.INFIX
    jobs["m"] = rng.integers(0, 200, count)
    which = np.arange(count) % texts
    jobs["n"] = text + which % 2
    jobs["t_off"] = which * (text + 1)
    jobs["p_off"] = texts * (text + 1) + np.concatenate([[0], np.cumsum(jobs["m"])[:-1]])
    plan = check(jobs)
    packed = 16 * plan["pool_words"]
    there = texts * (text + 1) + int(jobs["m"].sum())
    if text >= 4096:
        assert packed <= 2 * there + 16 * (plan["sequences"] + 512)
    if text >= 4096 and count > 20 * texts:
        assert plan["sequences"] <= count + texts


@pytest.mark.parametrize("scores", [(0, 0, 1, 0), (2, 4, 4, 2)])
def test_longest_sequences(check, scores):
    """Sequences whose row steps (or scores) would pass 32 bits stay off the anti-diagonal kernel,
    also where every step scores zero."""
    from spearfish_gb300 import batch as B
    for mode in (R.GLOBAL, R.PREFIX):
        rows = [dict(m=m, n=m, band=20, kind=B.JOB_AFFINE, mode=mode) for m in (1 << 20, (1 << 30) + 5)]
        kinds = check(_jobs(rows), [scores])["kinds"]
        assert kinds[0].startswith("wave16") and not kinds[1].startswith("wave16"), kinds


@pytest.mark.parametrize("mode", [R.INFIX, R.PREFIX, R.GLOBAL])
def test_caps_that_stop_pairs(check, mode):
    """A capped Global or Prefix pair may stop early where the kernel's column scores, 32 bits,
    hold its cap; caps of 2^30 and more (texts of more than 2^30 columns) never do."""
    from spearfish_gb300 import batch as B
    for n, k in ((900, 0), (900, 1799), (900, 1800), (1500000000, (1 << 30) - 1), (1500000000, 1 << 30),
                 (1500000000, 1200000000), (900, 0xFFFFFFFF)):
        plan = check(_jobs([dict(m=900, n=n, kind=B.JOB_MYERS, mode=mode, k=k)]))
        assert plan["myers_kcut"] == (mode != R.INFIX and k < 900 + n and k < 1 << 30), (n, k)


@pytest.mark.parametrize("passes,shared", [(644, False), (644, True), (2900, False), (20000, False)])
def test_streams_of_launches(check, passes, shared):
    """Few passes, not in a server: up to twelve launches on streams of their own.  The first launch
    starts before the others only while it leaves schedulers empty."""
    from spearfish_gb300 import batch as B
    odd = ((1, 3, 5, 2),)  # on the row kernels, a launch a class
    rows = [dict(m=900, n=900, band=20 + 640 * (q % 14) // 14, kind=B.JOB_AFFINE, mode=R.GLOBAL, want_cigar=1)
            for q in range(passes)]
    launches = check(_jobs(rows), odd, shared=shared)["launches"]
    streams = [x["stream"] for x in launches]
    assert 9 < len(launches) <= 16
    if passes <= 20 * 152 and not shared:
        assert len(set(streams)) == min(12, len(launches))
    else:
        assert max(streams) < 9
    assert [x["lead"] for x in launches] == [launches[0]["warps"] <= 4 * 152] + [False] * (len(launches) - 1)


@pytest.mark.parametrize("m", [60, 150, 363, 700, 1000])
@pytest.mark.parametrize("pairs", [1, 608, 609, 1500, 3000, 4500, 20000])
def test_pairs_that_share_a_warp(check, pairs, m):
    """Myers pairs share a warp as soon as each warp has a scheduler of its own, as far as its lanes
    hold them."""
    from spearfish_gb300 import batch as B
    plan = check(_jobs([dict(m=m, n=m + 100, kind=B.JOB_MYERS, mode=R.INFIX)] * pairs))
    (bucket,), (launch,) = plan["plan"]["buckets"], plan["launches"]
    share = min(32 // bucket["lanes"], -(-pairs // 608))
    assert launch["tasks"] == -(-pairs // share), (bucket, launch)


@pytest.mark.parametrize("longest", [40, 99, 100, 250])
@pytest.mark.parametrize("count", [1, 1200, 5000])
def test_few_short_prefix_passes(check, count, longest):
    """Few Prefix passes without traceback, all of short patterns, run on one kernel (the rows);
    with a long one among them, or many, each where it takes less time."""
    from spearfish_gb300 import batch as B
    rows = [dict(m=longest if q == 0 else 5 + q % 36, n=90, band=16, kind=B.JOB_EXTEND_WINDOW, mode=R.PREFIX,
                 window=90, xdrop=50, want_cigar=0) for q in range(count)]
    rows[0]["n"] = rows[0]["window"] = longest + 20
    plan = check(_jobs(rows))
    if count <= 3040 and longest < 100:
        assert set(plan["kinds"]) == {"affine16"}, set(plan["kinds"])
    else:
        assert "wave16x" in plan["kinds"]
    assert plan["strays"] == 0
