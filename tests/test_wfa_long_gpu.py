"""aw_set_wfa_long(0) starts every pair on one warp, also a call of a few long pairs."""
import numpy as np
import pytest

from anchorwave_b200 import wfa
from anchorwave_b200 import workloads as W

pytestmark = pytest.mark.gpu
PEN = (4, 4, 2, 24, 1)


@pytest.mark.parametrize("n,singletrack", [(1, False), (3, False), (1, True)])
def test_few_long_pairs_on_warps(gpu, restatement, n, singletrack):
    rng = np.random.default_rng(n)
    pairs = [W.divergent_pair(rng, 4200, 0.01, 0.01, 4.0) for _ in range(n)]
    ps, ts = [W.to_ascii(t) for _, t in pairs], [W.to_ascii(q) for q, _ in pairs]
    want = [restatement.wfa_align(p, t, *PEN, singletrack, memory_mode=0) for p, t in zip(ps, ts)]
    al = wfa.WfaAligner(*PEN, singletrack=singletrack, max_memory_abort=4 << 30)
    try:
        first, _ = al.align_batch(ps, ts)
        assert al.launches()[1] == 1  # by default they start on the cluster kernel
        wfa.set_long(0)
        wfa.set_wide(8192, 8192, 8)   # no hand-over below this width, which 1% does not reach
        on_warps, _ = al.align_batch(ps, ts)
        launches = al.launches()
    finally:
        wfa.set_wide(8192, 1024, 8)
        wfa.set_long(800)
        al.close()
    assert launches == (1, 0, 0)
    assert [r == w for r, w in zip(first, want)] == [True] * n
    assert [r == w for r, w in zip(on_warps, want)] == [True] * n
