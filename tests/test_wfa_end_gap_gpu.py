"""Pairs that end a few scores after a gap has run past the end of a sequence, on a score whose
predecessors are null (nothing can cost them): their headers are read by the backtrace."""
import numpy as np
import pytest

from anchorwave_b200 import wfa
from anchorwave_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _pairs(seed, n):
    rng = np.random.default_rng(seed)
    ps, ts = [], []
    for i in range(n):
        t = rng.integers(0, 4, int(rng.integers(410, 700))).astype(np.uint8)
        g, h = int(rng.integers(0, 7)), int(rng.integers(0, 4))
        q = t[h:len(t) - g].copy()
        at = rng.integers(0, len(q), int(rng.integers(0, 4)))
        q[at] = (q[at] + 1) & 3
        a, b = (t, q) if i % 2 else (q, t)
        ps.append(W.to_ascii(a))
        ts.append(W.to_ascii(b))
    return ps, ts


@pytest.mark.parametrize("pen", [(4, 4, 2, 24, 1), (4, 6, 2, 24, 2), (6, 8, 2, 75, 1), (9, 14, 5, 60, 3), (20, 30, 7, 90, 5)])
@pytest.mark.parametrize("singletrack,mode", [(False, 0), (True, 0), (False, 1)])
def test_short_scores(gpu, restatement, singletrack, mode, pen):
    ps, ts = _pairs(sum(pen), 240)
    want = [restatement.wfa_align(p, t, *pen, singletrack, memory_mode=mode) for p, t in zip(ps, ts)]
    rng = np.random.default_rng(1)
    dirty = [W.divergent_pair(rng, 1500, 0.1, 0.1, 4.0) for _ in range(300)]
    al = wfa.WfaAligner(*pen, singletrack=singletrack, memory_mode=mode, max_memory_abort=1 << 30)
    try:
        # CTAs of both sizes, then clusters; the pool holds what other pairs have left in it
        for width, n in ((8192, 240), (8192, 1), (1, 24), (1, 1)):
            wfa.set_wide(width, min(width, 1024), 8)
            al.align_batch([W.to_ascii(t) for _, t in dirty], [W.to_ascii(q) for q, _ in dirty])
            for at in range(0, 240 if n > 1 else 12, n):
                got, _ = al.align_batch(ps[at:at + n], ts[at:at + n])
                bad = [at + k for k, r in enumerate(got) if r != want[at + k]]
                assert not bad, (width, n, bad[:5])
    finally:
        wfa.set_wide(8192, 1024, 8)
        al.close()
