"""A full-width pair that stops at the deadline reports the ends as far as it got."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tlen", [100, 600])
def test_stopped_pair_reports_its_last_column(gpu, tlen):
    rng = np.random.default_rng(tlen)
    t = rng.integers(0, 4, tlen).astype(np.uint8)
    q = rng.integers(0, 4, 6_000_000).astype(np.uint8)
    mat = oracle.anchorwave_matrix(-4)
    run = lambda: gpu.ksw_extd2_batch([q], [t], mat, 4, 2, 24, 1, flag=0x01)[0]
    whole = run()
    assert not whole.stopped and whole.mte_q >= 0
    try:
        gpu.set_deadline(0.25)  # the sweep of six million rows takes over a second
        r = run()
    finally:
        gpu.set_deadline(0)
    assert r.stopped and r.score == -0x40000000 and r.n_cigar == 0
    # the last column's best score comes early (its later rows only add gaps)
    assert (r.mte, r.mte_q) == (whole.mte, whole.mte_q) and r.mqe_t == -1
