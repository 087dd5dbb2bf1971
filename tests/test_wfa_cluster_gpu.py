"""The cluster kernel's open and trimmed scores against the oracle restatement: pairs whose
wavefronts run past the end of a sequence early (overhangs, unrelated sequences), scores that
are null between others (penalties with a common factor), sequences with other letters than
ACGT, and clusters of both sizes (one pair, and more pairs than large clusters)."""
import numpy as np
import pytest

from anchorwave_b200 import wfa
from anchorwave_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _pairs(seed):
    rng = np.random.default_rng(seed)
    bases = lambda n: rng.integers(0, 4, n).astype(np.uint8)
    out = []
    for length, d in ((900, 0.05), (1500, 0.2), (2600, 0.1)):
        q, t = W.divergent_pair(rng, length, d, d, 4.0)
        out.append((q, t))
    q, t = out[0]
    out.append((q, np.concatenate([t, bases(600)])))                 # overhang at the end
    out.append((np.concatenate([bases(500), q]), t))                 # and at the start
    out.append((np.concatenate([q, bases(300)]), np.concatenate([bases(300), t])))
    out.append((bases(500), bases(900)))                             # unrelated
    out.append((bases(5), bases(1200)))                              # hardly a pattern
    n = out[1][0].copy()
    n[[3, 400, len(n) - 1]] = 4
    out.append((n, out[1][1]))
    return [W.to_ascii(t) for _, t in out], [W.to_ascii(q) for q, _ in out]


@pytest.mark.parametrize("pen", [(4, 4, 2, 24, 1), (4, 6, 2, 24, 2), (1, 1, 1, 3, 1), (3, 2, 4, 40, 3)])
@pytest.mark.parametrize("singletrack", [False, True])
def test_cluster_scores(gpu, restatement, singletrack, pen):
    ps, ts = _pairs(11)
    want = [restatement.wfa_align(p, t, *pen, singletrack, memory_mode=0) for p, t in zip(ps, ts)]
    al = wfa.WfaAligner(*pen, singletrack=singletrack, memory_mode=0, max_memory_abort=2 << 30)
    try:
        for clusters in (8, 7, 1):
            wfa.set_wide(1, 1, clusters)
            many, _ = al.align_batch(ps * 2, ts * 2)
            assert al.launches()[1] >= 1
            for i, r in enumerate(many):
                assert r == want[i % len(want)], (clusters, i)
            for i in (2, 3, 4, 7, 8):
                one, _ = al.align_batch(ps[i:i + 1], ts[i:i + 1])
                assert one[0] == want[i], (clusters, i)
    finally:
        wfa.set_wide(8192, 1024, 8)
        al.close()


@pytest.mark.parametrize("pen", [(4, 4, 2, 24, 1), (4, 6, 2, 24, 2), (6, 8, 2, 75, 1)])
@pytest.mark.parametrize("singletrack", [False, True])
def test_cta_scores(gpu, restatement, singletrack, pen):
    """The same pairs on CTAs of both sizes (few pairs, then many) and on warps."""
    ps, ts = _pairs(12)
    want = [restatement.wfa_align(p, t, *pen, singletrack, memory_mode=0) for p, t in zip(ps, ts)]
    al = wfa.WfaAligner(*pen, singletrack=singletrack, memory_mode=0, max_memory_abort=2 << 30)
    try:
        wfa.set_wide(0, 0, 8)
        for long_sum in (1, 1536, 0):
            wfa.set_long(long_sum)
            for times in (1, 80):
                got, _ = al.align_batch(ps * times, ts * times)
                for i, r in enumerate(got):
                    assert r == want[i % len(want)], (long_sum, times, i)
    finally:
        wfa.set_wide(8192, 1024, 8)
        wfa.set_long(800)
        al.close()


def test_cluster_beyond_shared_memory(gpu, restatement):
    """Sequences too long for the cluster kernel's shared memory: extended from global memory."""
    rng = np.random.default_rng(5)
    t = rng.integers(0, 4, 210_000).astype(np.uint8)
    q = np.delete(t, rng.integers(0, len(t), 12))
    at = rng.integers(0, len(q), 30)
    q[at] = (q[at] + 1) & 3
    p, x = W.to_ascii(t), W.to_ascii(q)
    al = wfa.WfaAligner(4, 4, 2, 24, 1, singletrack=True, max_memory_abort=2 << 30)
    try:
        wfa.set_wide(1, 1, 8)
        (got,), _ = al.align_batch([p], [x])
        assert al.launches()[1] == 1
    finally:
        wfa.set_wide(8192, 1024, 8)
        al.close()
    assert got == restatement.wfa_align(p, x, 4, 4, 2, 24, 1, True, memory_mode=0)
