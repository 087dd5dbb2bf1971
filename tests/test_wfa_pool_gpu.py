"""WFA pairs on whole CTAs in a pool that is too small for all of them at once: the next ones live on
the chunks of those that are finished, the ones that find the pool exhausted run again in later
rounds, with unchanged results."""
import numpy as np
import pytest

from anchorwave_b200 import wfa
from anchorwave_b200 import workloads as W

pytestmark = pytest.mark.gpu
PEN = (4, 4, 2, 24, 1)


def _pairs(seed, lengths, d):
    rng = np.random.default_rng(seed)
    pairs = [W.divergent_pair(rng, length, d, d, 4.0) for length in lengths]
    return [W.to_ascii(t) for _, t in pairs], [W.to_ascii(q) for q, _ in pairs]


@pytest.mark.parametrize("mode", [1, 2])
def test_pool_exhausted_inside_cta_pairs(gpu, restatement, mode):
    ps, ts = _pairs(5 + mode, [3000] * 56 + [1200] * 40, 0.12)
    al = wfa.WfaAligner(*PEN, memory_mode=mode, max_memory_abort=64 << 20)
    try:
        res, _ = al.align_batch(ps, ts)
        launches = al.launches()[0]
    finally:
        al.close()
    assert launches > 2  # one round takes two launches at most
    for i, (p, t, r) in enumerate(zip(ps, ts, res)):
        assert r == restatement.wfa_align(p, t, *PEN, False, memory_mode=mode), i


@pytest.mark.parametrize("length,d,singletrack,mode", [(8681, 0.04, False, 0), (1494, 0.25, False, 0),
                                                       (3336, 0.25, True, 0), (3774, 0.25, False, 1)])
def test_pair_that_takes_the_last_of_the_pool(gpu, restatement, length, d, singletrack, mode):
    """A pair alone in a pool that holds its trimmed wavefronts and little more, among pairs that
    share the same pool before and after it."""
    rng = np.random.default_rng(1)
    q, t = W.divergent_pair(rng, length, d, d, 4.0)
    p, x = W.to_ascii(t), W.to_ascii(q)
    few, fex = _pairs(3, [900] * 12, 0.05)
    al = wfa.WfaAligner(*PEN, singletrack=singletrack, memory_mode=mode, max_memory_abort=64 << 20)
    try:
        alone, _ = al.align_batch([p], [x])
        batch, _ = al.align_batch(few[:6] + [p] + few[6:], fex[:6] + [x] + fex[6:])
    finally:
        al.close()
    want = restatement.wfa_align(p, x, *PEN, singletrack, memory_mode=mode)
    assert want[0] == 0
    same = [alone[0] == want, batch[6] == want]
    same += [r == restatement.wfa_align(few[i], fex[i], *PEN, singletrack, memory_mode=mode)
             for i, r in enumerate(batch[:6] + batch[7:])]
    assert all(same), (same, alone[0][:2], batch[6][:2])


@pytest.mark.parametrize("singletrack,mode", [(False, 0), (True, 0)])
def test_finished_pairs_give_their_chunks_back(gpu, restatement, singletrack, mode):
    """4,000 pairs that take twice the pool and more together, a third of it at a time: one round (two
    launches at most), which takes as many more as the pool is short of if the chunks do not come back."""
    pool = 2000 << 20
    ps, ts = _pairs(31, [900] * 4000, 0.12 if singletrack else 0.06)
    al = wfa.WfaAligner(*PEN, singletrack=singletrack, memory_mode=mode, max_memory_abort=pool)
    try:
        wfa.set_wide(0, 0, 8)
        res, _ = al.align_batch(ps, ts)
        launches, total = al.launches()[0], al.memory()[1]
    finally:
        wfa.set_wide(8192, 1024, 8)
        al.close()
    assert all(r[0] == 0 for r in res)
    assert total > 2 * pool and launches <= 2, (launches, total)
    for i in range(0, len(ps), 100):
        assert res[i] == restatement.wfa_align(ps[i], ts[i], *PEN, singletrack, memory_mode=mode), i
