"""Short-lived clusters: the pair that each launch of the cluster kernel starts with, at every
cluster size, over many launches."""
import numpy as np
import pytest

from anchorwave_b200 import wfa
from anchorwave_b200 import workloads as W

pytestmark = pytest.mark.gpu
PEN = (4, 4, 2, 24, 1)


@pytest.mark.parametrize("clusters", [8, 5, 2, 1])
def test_many_launches(gpu, restatement, clusters):
    rng = np.random.default_rng(clusters)
    pairs = [W.divergent_pair(rng, length, 0.2, 0.2, 4.0) for length in (40, 90, 300)]
    ps, ts = [W.to_ascii(t) for _, t in pairs], [W.to_ascii(q) for q, _ in pairs]
    want = [restatement.wfa_align(p, t, *PEN, False, memory_mode=0) for p, t in zip(ps, ts)]
    al = wfa.WfaAligner(*PEN, max_memory_abort=1 << 30)
    try:
        wfa.set_wide(1, 1, clusters)
        for i in range(60):
            k = i % 3
            (got,), _ = al.align_batch(ps[k:k + 1], ts[k:k + 1])
            assert al.launches()[1] == 1
            assert got == want[k], i
    finally:
        wfa.set_wide(8192, 1024, 8)
        al.close()
