"""The memory figure of an alignment, by which a caller may refuse it: what the pair holds, about
the same on a warp, a CTA or a cluster."""
import numpy as np
import pytest

from anchorwave_b200 import wfa
from anchorwave_b200 import workloads as W

pytestmark = pytest.mark.gpu
PEN = (4, 4, 2, 24, 1)
CHUNK = 256 << 10


@pytest.mark.parametrize("singletrack,mode", [(False, 0), (True, 0), (False, 1), (False, 2)])
@pytest.mark.parametrize("length,d", [(300, 0.05), (4000, 0.02), (6000, 0.04)])
def test_figure_does_not_depend_on_the_kernel(gpu, length, d, singletrack, mode):
    rng = np.random.default_rng(length)
    q, t = W.divergent_pair(rng, length, d, d, 4.0)
    p, x = W.to_ascii(t), W.to_ascii(q)
    al = wfa.WfaAligner(*PEN, singletrack=singletrack, memory_mode=mode, max_memory_abort=8 << 30)
    figures = {}
    try:
        # by default (few long pairs: a cluster in high memory), a CTA, a warp
        for name, width, long_sum in (("default", 8192, 800), ("cta", 0, 800), ("warp", 0, 0)):
            wfa.set_wide(width, min(width, 1024), 8)
            wfa.set_long(long_sum)
            (res,), _ = al.align_batch([p], [x])
            assert res[0] == 0
            figures[name] = al.memory()[0]
    finally:
        wfa.set_wide(8192, 1024, 8)
        wfa.set_long(800)
        al.close()
    warp = figures["warp"]
    # wavefronts are stored untrimmed there (a few diagonals a side); in the piggyback modes each of a
    # CTA's warps reserves blocks of its own, which at four warps took five chunks
    spare = 5 * CHUNK if mode else CHUNK
    for name in ("default", "cta"):
        assert warp // 2 <= figures[name] <= 1.05 * warp + spare, figures
