"""A plan that exists follows aw_set_tuning: the strips of its long pairs on a warp each, or all
strips of a pair on one warp, which takes many times as long when the pairs are few."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def test_plan_follows_large_warps(gpu, restatement):
    rng = np.random.default_rng(9)
    ts = [rng.integers(0, 4, 20_000 - 64 * i).astype(np.uint8) for i in range(64)]
    qs = []
    for t in ts:
        q = t.copy()
        at = rng.random(len(t)) < 0.05
        q[at] = rng.integers(0, 4, int(at.sum()))
        qs.append(q)
    mat = oracle.anchorwave_matrix(-4)
    plan = gpu.KswPlan(qs, ts, mat, 4, 2, 24, 1, flag=0x01)
    plan.upload()
    times, keys = {}, {}
    try:
        for warps in (8, 8, 8, 1, 1, 4, 4):  # eager, captured and replayed; captured anew at each change
            gpu.set_tuning(warps, 4096)
            times.setdefault(warps, []).append(plan.execute())
            keys[warps] = [r.key() for r in plan.download()]
    finally:
        gpu.set_tuning(8, 4096)
        plan.close()
    assert keys[1] == keys[8] and keys[4] == keys[8]
    assert keys[8][0] == restatement.ksw_extd2(qs[0].tobytes(), ts[0].tobytes(), mat, 4, 2, 24, 1, flag=0x01).key()
    assert min(times[1]) > 3 * max(min(times[8]), min(times[4])), times
