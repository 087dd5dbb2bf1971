"""The traceback walks' runs, tiles and gap searches at their edges: gaps and diagonal runs
of one warp's width and one tile's width, one more and one less, long gaps in both
directions, and walks that end on either matrix edge, against the oracle restatement."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
ST = 0x1000


def _gapped(rng, lengths, run):
    """A target and a query that differ by gaps of the given lengths (positive: deleted from
    the query, negative: inserted into it), `run` equal bases apart."""
    t, q = [], []
    for k in lengths:
        same = rng.integers(0, 4, run)
        extra = rng.integers(0, 4, abs(k))
        t += [same] + ([extra] if k > 0 else [])
        q += [same] + ([extra] if k < 0 else [])
    tail = rng.integers(0, 4, run)
    return np.concatenate(q + [tail]).astype(np.uint8), np.concatenate(t + [tail]).astype(np.uint8)


def _cases():
    rng = np.random.default_rng(8)
    edges = [1, -1, 2, 15, -16, 17, -31, 32, -33, 33, -32, 31, 63, -64, 65, -63, 64, -65]
    out = [_gapped(rng, edges, run) for run in (31, 32, 33, 64)]
    out += [_gapped(rng, [k], 80) for k in (500, -500, 129, -127)]
    # gaps at either end, and one sequence much longer than the other
    out.append((out[0][0][100:], out[0][1]))
    out.append((out[0][0], out[0][1][100:]))
    out.append((out[1][0][:40], out[1][1]))
    out.append((out[1][0], out[1][1][:40]))
    return out


@pytest.mark.parametrize("columns", [8, 4])
@pytest.mark.parametrize("flag,band", [(0, None), (0, 600), (ST, None), (ST, 600)])
def test_walk_edges(gpu, restatement, flag, band, columns):
    pairs = _cases()
    mat = oracle.anchorwave_matrix(-4)
    ws = [-1 if band is None else max(band, abs(len(q) - len(t)) + 40) for q, t in pairs]
    gpu.set_band_columns(columns)
    try:
        res = gpu.ksw_extd2_batch([q for q, _ in pairs], [t for _, t in pairs], mat, 4, 2, 24, 1, w=ws, flag=flag)
    finally:
        gpu.set_band_columns(0)
    for (q, t), w, r in zip(pairs, ws, res):
        o = restatement.ksw_extd2(q.tobytes(), t.tobytes(), mat, 4, 2, 24, 1, w=w, flag=flag)
        assert r.key() == o.key(), (len(q), len(t), w)
