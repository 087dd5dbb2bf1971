"""The WFA kernels' groups of threads against the oracle restatement: pairs on warps, on whole
CTAs of both sizes (few pairs, or one long pair among many), in the cluster kernel, and in a
pool small enough that pairs live on the chunks that finished pairs gave back."""
import numpy as np
import pytest

from anchorwave_b200 import wfa
from anchorwave_b200 import workloads as W

pytestmark = pytest.mark.gpu
MODES = [(False, 0), (True, 0), (False, 1), (False, 2)]


def _pairs(seed, lengths, dmax):
    rng = np.random.default_rng(seed)
    ps, ts = [], []
    for i, length in enumerate(lengths):
        q, t = W.divergent_pair(rng, length, 0.0, dmax, 4.0)
        if i % 6 == 0:
            q = q.copy()
            q[rng.integers(0, len(q), 2)] = 4
        ps.append(W.to_ascii(t))
        ts.append(W.to_ascii(q))
    return ps, ts


def _check(restatement, pen, ps, ts, singletrack, mode, res):
    for i, (p, t, r) in enumerate(zip(ps, ts, res)):
        assert r == restatement.wfa_align(p, t, *pen, singletrack, memory_mode=mode), (i, len(p), len(t))


@pytest.mark.parametrize("pen", [(4, 4, 2, 24, 1), (6, 8, 2, 75, 1), (3, 2, 3, 40, 2)])
@pytest.mark.parametrize("singletrack,mode", MODES)
def test_groups(gpu, restatement, singletrack, mode, pen):
    ps, ts = _pairs(7 + mode, [1, 2, 31, 100, 700, 760, 800, 1500, 2500, 4000], 0.1)
    al = wfa.WfaAligner(*pen, singletrack=singletrack, memory_mode=mode, max_memory_abort=4 << 30)
    try:
        first, _ = al.align_batch(ps, ts)
        _check(restatement, pen, ps, ts, singletrack, mode, first)
        for long_sum, width in ((0, 0), (1, 0), (1, 64), (1536, 8192)):
            wfa.set_long(long_sum)
            wfa.set_wide(width, min(width, 64), 8)
            got, _ = al.align_batch(ps, ts)
            assert got == first, (long_sum, width)
    finally:
        wfa.set_long(1536)
        wfa.set_wide(8192, 1024, 8)
        al.close()


@pytest.mark.parametrize("singletrack,mode", MODES)
def test_one_long_pair_among_many(gpu, restatement, singletrack, mode):
    lengths = [5000] + [800] * 60 + [60] * 300
    ps, ts = _pairs(3 + mode, lengths, 0.05)
    al = wfa.WfaAligner(4, 4, 2, 24, 1, singletrack=singletrack, memory_mode=mode, max_memory_abort=4 << 30)
    res, _ = al.align_batch(ps, ts)
    al.close()
    _check(restatement, (4, 4, 2, 24, 1), ps, ts, singletrack, mode, res)


@pytest.mark.parametrize("singletrack,mode", MODES)
def test_pool_chunks_are_reused(gpu, restatement, singletrack, mode):
    """600 pairs that take about 1.3 MB each in high memory, in a pool of 160 MB: one round
    suffices once the chunks of finished pairs serve the next ones."""
    ps, ts = _pairs(21 + mode, [900] * 600, 0.06)
    al = wfa.WfaAligner(4, 4, 2, 24, 1, singletrack=singletrack, memory_mode=mode, max_memory_abort=160 << 20)
    res, _ = al.align_batch(ps, ts)
    al.close()
    _check(restatement, (4, 4, 2, 24, 1), ps, ts, singletrack, mode, res)
