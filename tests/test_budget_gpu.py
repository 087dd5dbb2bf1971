"""Traceback budgets that just hold a batch: nothing that fits is refused."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
ST = 0x1000


# pairs, length, band, and a budget that holds the tracks (two bytes a cell of the strips' rows, and
# 31 rows of skew) and the boundary columns (eight bytes a row) of strips of 128 or of 256 columns
@pytest.mark.parametrize("n,length,w,budget", [(1, 100, 20, 34560), (1, 700, 64, 509184), (16, 2000, 200, 3593216),
                                               (3, 9000, 700, 31223040)])
def test_banded_singletrack_within_budget(gpu, restatement, n, length, w, budget):
    rng = np.random.default_rng(length)
    ts = [rng.integers(0, 4, length).astype(np.uint8) for _ in range(n)]
    qs = []
    for t in ts:
        q = t.copy()
        at = rng.random(length) < 0.05
        q[at] = rng.integers(0, 4, int(at.sum()))
        qs.append(q)
    mat = oracle.anchorwave_matrix(-4)
    try:
        gpu.set_traceback_budget(budget)
        res = gpu.ksw_extd2_batch(qs, ts, mat, 4, 2, 24, 1, w=[w] * n, flag=ST)
    finally:
        gpu.set_traceback_budget(0)
    for q, t, r in zip(qs, ts, res):
        assert r.key() == restatement.ksw_extd2(q.tobytes(), t.tobytes(), mat, 4, 2, 24, 1, w=w, flag=ST).key()


def _device_bytes(gpu, call):
    import torch
    gpu.release_thread_buffers()
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    res = call()
    used = free - torch.cuda.mem_get_info()[0]
    gpu.release_thread_buffers()
    return used, res


@pytest.mark.parametrize("length,score_only,budget", [(60_000, True, 64 << 20), (9000, False, 82 << 20)])
def test_full_matrix_boundary_columns_within_budget(gpu, restatement, length, score_only, budget):
    """One pair, whose narrow strips (eight bytes a row for 128 columns) would exceed the budget, with
    the traceback in the second case: wide strips are used, and the results are the same."""
    rng = np.random.default_rng(length)
    t = rng.integers(0, 4, length).astype(np.uint8)
    q = t.copy()
    at = rng.random(length) < 0.05
    q[at] = rng.integers(0, 4, int(at.sum()))
    mat = oracle.anchorwave_matrix(-4)
    run = lambda: gpu.ksw_extd2_batch([q], [t], mat, 4, 2, 24, 1, flag=0x01 if score_only else 0)
    _, free_choice = _device_bytes(gpu, run)
    try:
        gpu.set_traceback_budget(budget)
        used, (res,) = _device_bytes(gpu, run)
    finally:
        gpu.set_traceback_budget(0)
    assert res.key() == free_choice[0].key()
    # beside the two arenas: sequences, CIGAR slots and records, and 2 MiB pages of each buffer
    assert used <= budget + 24 * length + (48 << 20), used
