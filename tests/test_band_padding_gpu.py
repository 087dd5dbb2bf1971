"""Narrow bands whose computed blocks reach far beyond the band, under penalties that let the
values of the cells out there grow large (by q + e - e2 an anti-diagonal: past 16-bit fields of
the sweep, and under the last two sets within its last 16-column block already), against the
oracle restatement."""
import numpy as np
import pytest

import oracle
from anchorwave_b200 import ksw2

pytestmark = pytest.mark.gpu
RIGHT, GENERIC, ST, SSE_ST, SCORE_ONLY = 0x02, 0x04, 0x1000, 0x4000, 0x01
PEN = [(4, 2, 24, 1), (16, 2, 41, 1), (10, 9, 40, 1), (12, 12, 30, 1), (30, 4, 40, 1), (46, 2, 47, 1), (44, 3, 46, 1)]
MISMATCH = [-4, -9, -30, -10, -20, -2, -5]


def _pair(rng, kind):
    n = int(rng.integers(60, 420))
    bases = lambda k: rng.integers(0, 2 if kind == 4 else 4, k).astype(np.uint8)
    t = bases(n)
    q = t.copy()
    if kind == 1:
        q = bases(n)
    elif kind == 2:
        at, k = int(rng.integers(0, n // 2)), int(rng.integers(1, n // 3))
        q = np.concatenate([q[:at], q[at + k:]])
    elif kind == 3:
        at, k = int(rng.integers(0, n // 2)), int(rng.integers(1, n // 3))
        q = np.concatenate([q[:at], bases(k), q[at:]])
    sub = rng.random(len(q)) < rng.uniform(0, 0.4)
    q[sub] = bases(int(sub.sum()))
    return q, t, max(1, abs(len(q) - len(t))) + int(rng.integers(0, 24))


def _matrix(mis):
    mat = np.full((5, 5), mis, np.int8)
    np.fill_diagonal(mat, 0)
    mat[4, :] = mat[:, 4] = -1
    return mat.tobytes()


@pytest.mark.parametrize("flag", [0, RIGHT, GENERIC, SCORE_ONLY, ST, ST | SSE_ST])
@pytest.mark.parametrize("pen,mis", list(zip(PEN, MISMATCH)))
def test_padding(gpu, restatement, pen, mis, flag):
    rng = np.random.default_rng(flag + pen[0])
    qs, ts, ws = zip(*[_pair(rng, i % 5) for i in range(1200 if pen[0] == 10 else 300)])
    mat = _matrix(mis)
    more = {"block": 16} if flag & SSE_ST else {}
    want = [restatement.ksw_extd2(q.tobytes(), t.tobytes(), mat, *pen, w=w, flag=flag & ~SSE_ST, **more).key()
            for q, t, w in zip(qs, ts, ws)]
    plan = ksw2.KswPlan(qs, ts, mat, *pen, w=ws, flag=flag)
    plan.upload()
    for _ in range(3):  # eager, captured, replayed
        plan.execute()
        got = [r.key() for r in plan.download()]
        bad = [(len(q), len(t), w) for q, t, w, g, k in zip(qs, ts, ws, got, want) if g != k]
        assert not bad, (len(bad), bad[:5])
    plan.close()


@pytest.mark.parametrize("pen,mis", list(zip(PEN, MISMATCH)))
def test_padding_in_recompute_rounds(gpu, restatement, pen, mis):
    """A traceback beyond the budget: recomputed in groups of strips, each with its own bytes."""
    rng = np.random.default_rng(pen[0])
    mat = _matrix(mis)
    t = rng.integers(0, 4, 3000).astype(np.uint8)
    q = np.concatenate([t[:700], t[760:1500], rng.integers(0, 4, 90).astype(np.uint8), t[1500:]])
    sub = rng.random(len(q)) < 0.2
    q[sub] = rng.integers(0, 4, int(sub.sum()))
    ws = [31, 33, 48, 64, 100]
    try:
        gpu.set_traceback_budget(150_000)
        res = gpu.ksw_extd2_batch([q] * 5, [t] * 5, mat, *pen, w=ws)
    finally:
        gpu.set_traceback_budget(0)
    for w, r in zip(ws, res):
        assert r.key() == restatement.ksw_extd2(q.tobytes(), t.tobytes(), mat, *pen, w=w).key(), w


@pytest.mark.parametrize("pen", [(0, 1, 5, 1), (2, 2, 60, 2), (20, 1, 70, 1), (4, 2, 24, 1)])
@pytest.mark.parametrize("flag", [0, RIGHT, SCORE_ONLY, ST, ST | SSE_ST])
def test_narrowest_bands(gpu, restatement, pen, flag):
    """Bands of 0 to 3; with equal extensions a band of one tracks a maximum above zero."""
    rng = np.random.default_rng(pen[2] + flag)
    mat = _matrix(-1)
    qs, ts, ws = [], [], []
    for i in range(160):
        n = int(rng.integers(1, 40))
        t = rng.integers(0, 4, n).astype(np.uint8)
        q = np.concatenate([t, t[:1]])[int(rng.integers(0, 2)):n + int(rng.integers(0, 2))]
        qs.append(q if len(q) else t[:1])
        ts.append(t)
        ws.append(i % 4)
    res = gpu.ksw_extd2_batch(qs, ts, mat, *pen, w=ws, flag=flag)
    more = {"block": 16} if flag & SSE_ST else {}
    bad = [(len(q), len(t), w) for q, t, w, r in zip(qs, ts, ws, res)
           if r.key() != restatement.ksw_extd2(q.tobytes(), t.tobytes(), mat, *pen, w=w, flag=flag & ~SSE_ST, **more).key()]
    assert not bad, (len(bad), bad[:5])
