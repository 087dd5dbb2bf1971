"""The banded kernel's edge steps where their closed forms change: band widths around the
SIMD blocks (the score fill's length rounds w and w + 1 up to 16), lengths around the strip
widths, and length differences that move the last rows' rule, against the oracle restatement."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
GENERIC, ST, SSE_ST, SCORE_ONLY = 0x04, 0x1000, 0x4000, 0x01


def _pair(rng, tlen, diff):
    t = rng.integers(0, 4, tlen).astype(np.uint8)
    q = t.copy()
    sub = rng.random(tlen) < 0.08
    q[sub] = rng.integers(0, 4, int(sub.sum()))
    at = int(rng.integers(1, max(2, tlen - abs(diff) - 1)))
    q = np.concatenate([q[:at], q[at + diff:]]) if diff > 0 else \
        np.concatenate([q[:at], rng.integers(0, 4, -diff).astype(np.uint8), q[at:]])
    return q, t


@pytest.mark.parametrize("columns", [8, 4])
@pytest.mark.parametrize("flag", [0, GENERIC, SCORE_ONLY, ST, ST | SSE_ST])
def test_edge_steps(gpu, restatement, flag, columns):
    rng = np.random.default_rng(flag + columns)
    qs, ts, ws = [], [], []
    for w in (14, 15, 16, 17, 31, 32, 33, 47, 63, 64, 65, 127, 128, 300):
        for tlen in (127, 128, 129, 255, 257, 511, 640):
            q, t = _pair(rng, tlen, int(rng.integers(-min(w, tlen // 2), min(w, tlen // 2) + 1)))
            qs.append(q)
            ts.append(t)
            ws.append(w)
    mat = oracle.anchorwave_matrix(-4)
    gpu.set_band_columns(columns)
    try:
        res = gpu.ksw_extd2_batch(qs, ts, mat, 4, 2, 24, 1, w=ws, flag=flag)
    finally:
        gpu.set_band_columns(0)
    more = {"block": 16} if flag & SSE_ST else {}
    bad = []
    for q, t, w, r in zip(qs, ts, ws, res):
        o = restatement.ksw_extd2(q.tobytes(), t.tobytes(), mat, 4, 2, 24, 1, w=w, flag=flag & ~SSE_ST, **more)
        if r.key() != o.key():
            bad.append((len(q), len(t), w))
    assert not bad, (len(bad), bad[:5])
