"""Both strip widths of the full-matrix kernel at their edges, against the oracle restatement:
few pairs run on narrow strips (128 columns), a batch with work enough for the GPU on wide
ones (512), whose strips go to one warp each or, with aw_set_tuning, to one warp per pair."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
RIGHT, SCORE_ONLY, SEMI, ST = 0x02, 0x01, 0x800, 0x1000
MAT = oracle.anchorwave_matrix(-4)


def _pair(rng, qlen, tlen):
    t = rng.integers(0, 4, tlen).astype(np.uint8)
    q = np.resize(t, qlen).copy()
    sub = rng.random(qlen) < 0.1
    q[sub] = rng.integers(0, 5, int(sub.sum()))
    return q, t


def _check(gpu, restatement, pairs, flag, picks):
    res = gpu.ksw_extd2_batch([q for q, _ in pairs], [t for _, t in pairs], MAT, 4, 2, 24, 1, flag=flag)
    for i in picks:
        q, t = pairs[i]
        o = restatement.ksw_extd2(q.tobytes(), t.tobytes(), MAT, 4, 2, 24, 1, flag=flag)
        assert res[i].key() == o.key(), (len(q), len(t), hex(flag))


@pytest.mark.parametrize("flag", [0, RIGHT, SCORE_ONLY, SEMI, ST])
def test_narrow_strips(gpu, restatement, flag):
    rng = np.random.default_rng(flag)
    pairs = [_pair(rng, q, t) for t in (1, 2, 3, 4, 127, 128, 129, 255, 257, 640) for q in (1, 7, 8, 62, 63, 64, 65, 300)]
    _check(gpu, restatement, pairs, flag, range(len(pairs)))


@pytest.mark.parametrize("warps", [8, 1])
@pytest.mark.parametrize("flag", [0, RIGHT, SCORE_ONLY, SEMI, ST])
def test_wide_strips(gpu, restatement, flag, warps):
    rng = np.random.default_rng(100 + flag)
    edges = [_pair(rng, q, t) for t in (1, 8, 9, 15, 16, 17, 511, 512, 513, 1024, 1025) for q in (1, 31, 63, 64, 500)]
    pairs = edges + [_pair(rng, 700, 512) for _ in range(1100)]
    gpu.set_tuning(large_warps=warps, large_tlen_threshold=4096)
    try:
        _check(gpu, restatement, pairs, flag, list(range(len(edges))) + list(range(len(edges), len(pairs), 90)))
    finally:
        gpu.set_tuning(large_warps=8, large_tlen_threshold=4096)
