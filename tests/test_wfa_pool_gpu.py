"""WFA pairs on whole CTAs in a pool that is too small for all of them at once: the ones that
find it exhausted run again in later rounds, with unchanged results."""
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
