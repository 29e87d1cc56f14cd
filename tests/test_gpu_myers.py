"""The Myers kernels (sf_myers.cu) against the oracle at the edges of their layout: patterns that
fill a lane's blocks or a pair's lanes exactly, miss by one base or pass by one; texts around the
chunks of 32 steps; teams of two and four warps up to the longest pattern; pairs of different
length side by side in a warp; every mode, with and without caps on either side of the distance.
Few pairs run one to a warp (or team), many run several to a warp: both are covered."""
import json

import numpy as np
import pytest

import oracle as O
import refcases as R

pytestmark = pytest.mark.gpu

NONE = 0xFFFFFFFF
# More pairs than this run several to a warp on any GPU this library is built for.
PACKED = 3400


@pytest.fixture(scope="module")
def ctx():
    from spearfish_gb300 import build
    build.build()
    from spearfish_gb300 import batch as B
    c = B.Context(0)
    yield c
    c.close()


def _run(ctx, rows):
    """rows: (pattern, text, mode, k).  Returns the distances and the (blocks, lanes) used."""
    from spearfish_gb300 import batch as B
    pb = B.PoolBuilder()
    jobs = B.new_jobs(len(rows))
    for j, (p, t, mode, k) in zip(jobs, rows):
        j["p_off"], j["m"], j["t_off"], j["n"] = pb.add(p), len(p), pb.add(t), len(t)
        j["kind"], j["mode"], j["k"] = B.JOB_MYERS, mode, k
    plan = B.Plan(ctx, jobs, pb.size)
    try:
        plan.upload(pb.build())
        plan.execute()
        got = plan.download().results["distance"].copy()
        plan.execute()
        assert np.array_equal(got, plan.download().results["distance"])
        used = {(b["c"], b["lanes"]) for b in json.loads(plan.describe())["buckets"]}
    finally:
        plan.close()
    return got, used


def _check(rows, got):
    for q, (p, t, mode, k) in enumerate(rows):
        want = O.myers_distance(p, t, mode, None if k == NONE else k) if k != NONE else \
            O.myers_distance(p, t, mode)
        assert int(got[q]) == (NONE if want is None else want), (q, len(p), len(t), mode, k)


def _pair(rng, m, n):
    """A pattern of m bases and a related text of n bases."""
    p = rng.integers(0, 4, m).astype(np.uint8)
    t = np.asarray(R.mutate(p.tolist(), R.rand_edits(rng, max(1, m // 12), m)), np.uint8) \
        if m else np.zeros(0, np.uint8)
    t = np.concatenate([t, rng.integers(0, 4, max(0, n - t.size)).astype(np.uint8)])[:n]
    return p, t


@pytest.mark.parametrize("packed", [False, True])
def test_block_and_chunk_edges(ctx, packed):
    rng = np.random.default_rng(2701 + packed)
    rows = []
    ms = [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 191, 193, 255, 257, 320, 511, 513, 639, 641,
          1023, 1024, 1025, 1343, 1345, 2047, 2048, 2049]
    ns = [0, 1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 97, 500]
    for m in ms:
        for n in (ns if m < 300 else (m - 3, m, m + 1, m + 32, 40)):
            mode = int(rng.integers(0, 3))
            rows.append((*_pair(rng, m, n), mode, NONE))
            d = O.myers_distance(*rows[-1][:2], mode)
            rows.append((*rows[-1][:2], mode, int(rng.choice([0, max(0, d - 1), d, d + 1]))))
    while packed and len(rows) < PACKED:
        m = int(np.exp(rng.uniform(0, np.log(700))))
        p, t = _pair(rng, m, int(m * rng.uniform(0.5, 1.5)) + 1)
        if rng.random() < 0.3:
            t = rng.integers(0, 4, t.size).astype(np.uint8)
        rows.append((p, t, int(rng.integers(0, 3)),
                     NONE if rng.random() < 0.4 else int(rng.integers(0, m + 2))))
    order = rng.permutation(len(rows))
    rows = [rows[i] for i in order]
    got, used = _run(ctx, rows)
    assert used >= ({(1, 32), (1, 16), (2, 17)} if packed else {(1, 1), (1, 2), (1, 32), (1, 64)})
    _check(rows, got)


def test_teams(ctx):
    """Two and four warps to a pair: 33 to 512 blocks, texts shorter than the warps' start, caps
    that stop a pair early, late or never."""
    rng = np.random.default_rng(2711)
    rows = []
    for m in (2049, 4095, 4096, 4097, 8191, 8193, 16384, 16385, 24577, 32768):
        for n in (1, 60, 190, 300, m - 40, m + 90):
            p, t = _pair(rng, m, n)
            mode = int(rng.integers(0, 3))
            rows.append((p, t, mode, NONE))
            rows.append((p, rng.integers(0, 4, n).astype(np.uint8), 2, m // 10))
            rows.append((p, t, 1 + n % 2, m // 5))
    got, used = _run(ctx, rows)
    assert used >= {(1, 64), (1, 128), (2, 128), (3, 128), (4, 128)}, used
    _check(rows, got)
