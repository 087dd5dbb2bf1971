"""Traceback budgets that just hold a batch: nothing that fits is refused."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
ST = 0x1000


# pairs, length, band, and a budget that holds the tracks (two bytes a cell of the strips' rows, and
# 31 rows of skew) and the boundary columns (eight bytes a row) of strips of 128 or of 256 columns
@pytest.mark.parametrize("n,length,w,budget", [(1, 100, 20, 34560), (1, 700, 64, 509184), (16, 2000, 200, 3593216),
                                               (3, 9000, 700, 31223040)])
def test_banded_singletrack_within_budget(gpu, restatement, n, length, w, budget):
    rng = np.random.default_rng(length)
    ts = [rng.integers(0, 4, length).astype(np.uint8) for _ in range(n)]
    qs = []
    for t in ts:
        q = t.copy()
        at = rng.random(length) < 0.05
        q[at] = rng.integers(0, 4, int(at.sum()))
        qs.append(q)
    mat = oracle.anchorwave_matrix(-4)
    try:
        gpu.set_traceback_budget(budget)
        res = gpu.ksw_extd2_batch(qs, ts, mat, 4, 2, 24, 1, w=[w] * n, flag=ST)
    finally:
        gpu.set_traceback_budget(0)
    for q, t, r in zip(qs, ts, res):
        assert r.key() == restatement.ksw_extd2(q.tobytes(), t.tobytes(), mat, 4, 2, 24, 1, w=w, flag=ST).key()
