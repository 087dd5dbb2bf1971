"""The work that users of this framework have it do, one measurable case each.

AnchorWave's alignment stage hands over intervals one at a time or in batches: KSW2 with a
CIGAR (full matrix, banded, Singletrack), the score-certified rescue, gap-affine-2p WFA in its
memory modes, the selector's pass over the sequences, and a serving loop that takes a mixed
stream.  A case is a dict of plain sizes; sequences are seeded synthetic intervals with the
shapes of ``anchorwave_b200.workloads``, so lengths within a case are ragged.
"""
import ctypes
import math

import numpy as np

from anchorwave_b200 import ksw2, selector, serve, wfa
from anchorwave_b200 import workloads as W

GIB = 1 << 30
# match 0, mismatch 4, gaps 4 + 2L and 24 + L: the scoring of the repository's workloads
MAT = ksw2.anchorwave_matrix(-4)
GAPS = (4, 2, 24, 1)
ANCHORWAVE_PENALTIES = (-4, -4, -2, -24, -1)
WFA_PENALTIES = (4, 4, 2, 24, 1)
TRACEBACK_BUDGET = 40 * GIB   # the program's -M envelope for KSW2 tracebacks
WFA_POOL = 20 * GIB           # each aligner's wavefront memory
SERVER_BUDGET = 16 * GIB      # device memory of a server

_MODES = {"standard": (False, wfa.WAVEFRONT_MEMORY_HIGH), "singletrack": (True, wfa.WAVEFRONT_MEMORY_HIGH),
          "medium": (False, wfa.WAVEFRONT_MEMORY_MED)}


def listed():
    return [
        # the smallest call: one short interval between two close anchors, latency only
        {"name": "ksw single 300 bp", "kind": "single", "lmin": 300, "lmax": 300, "deletion": 0},
        # an ordinary single call: one 5 kb interval with a 500 bp deletion
        {"name": "ksw single 5 kb", "kind": "single", "lmin": 5000, "lmax": 5000, "deletion": 500},
        # a chromosome's intervals in one submission, host buffers in, CIGARs out
        {"name": "ksw batch 0.2-20 kb", "kind": "batch", "n": 768, "lmin": 200, "lmax": 20000, "ambiguous": 0},
        # many short intervals, some with Ns (the generic scoring matrix)
        {"name": "ksw batch short", "kind": "batch", "n": 3001, "lmin": 50, "lmax": 1500, "ambiguous": 1},
        # long intervals with repeats and long indels, band of 10% of the shorter sequence
        {"name": "ksw banded long", "kind": "banded", "n": 4, "lmin": 60000, "lmax": 160000, "percent": 10},
        # the low-memory Singletrack traceback, unbanded, on mid-size intervals
        {"name": "ksw singletrack", "kind": "singletrack", "n": 128, "lmin": 2000, "lmax": 8000},
        # score-certified rescue: score-only optimum, then banded tracebacks until one reaches it
        {"name": "ksw certified", "kind": "certified", "n": 24, "lmin": 2000, "lmax": 20000, "band": 64,
         "band_max": 4000},
        # the batched WFA of low-divergence intervals, every wavefront kept
        {"name": "wfa batch", "kind": "wfa", "mode": "standard", "n": 4096, "lmin": 100, "lmax": 10000,
         "dmin": 0.005, "dmax": 0.05},
        # one long divergent interval, as the selector routes them to SingletrackWfa: latency
        {"name": "wfa long interval", "kind": "wfa", "mode": "singletrack", "n": 1, "lmin": 24000, "lmax": 24000,
         "dmin": 0.12, "dmax": 0.12},
        # the piggyback traceback, for batches whose wavefronts would not fit
        {"name": "wfa medium memory", "kind": "wfa", "mode": "medium", "n": 2048, "lmin": 100, "lmax": 10000,
         "dmin": 0.005, "dmax": 0.05},
        # the selector's pass over the sequences of a batch (sketches, composition, entropy)
        {"name": "selector pass", "kind": "selector", "n": 512, "lmin": 200, "lmax": 20000},
        # a mixed stream through the serving loop: WFA, full and banded KSW2, results in order
        {"name": "serving stream", "kind": "serve", "n": 512, "lmax": 40000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "batch", "banded", "singletrack", "certified", "wfa", "selector", "serve"])
    if kind == "single":
        length = _log_uniform(rng, 50, 20000)
        return {"kind": kind, "lmin": length, "lmax": length, "deletion": rng.choice([0, length // 10])}
    if kind == "batch":
        lmin = _log_uniform(rng, 50, 2000)
        lmax = _log_uniform(rng, 2 * lmin, 20000)
        most = min(3000, int(768 * 20000 ** 2 / lmax ** 2))
        return {"kind": kind, "n": _log_uniform(rng, 8, most), "lmin": lmin, "lmax": lmax,
                "ambiguous": rng.choice([0, 1])}
    if kind == "banded":
        lmin = _log_uniform(rng, 2000, 100000)
        return {"kind": kind, "n": _log_uniform(rng, 1, min(64, 400000 // lmin)), "lmin": lmin,
                "lmax": int(lmin * 1.6), "percent": rng.choice([2, 5, 10])}
    if kind == "singletrack":
        lmin = _log_uniform(rng, 100, 4000)
        return {"kind": kind, "n": _log_uniform(rng, 4, 128), "lmin": lmin, "lmax": 2 * lmin}
    if kind == "certified":
        lmin = _log_uniform(rng, 200, 8000)
        return {"kind": kind, "n": rng.randint(1, 24), "lmin": lmin, "lmax": _log_uniform(rng, lmin, 20000),
                "band": rng.choice([16, 64, 200]), "band_max": rng.choice([1000, 4000])}
    if kind == "wfa":
        mode = rng.choice(["standard", "singletrack", "medium"])
        if rng.random() < 0.3 and mode != "medium":
            length = _log_uniform(rng, 2000, 30000)
            d = rng.uniform(0.02, 0.12)
            return {"kind": kind, "mode": mode, "n": rng.randint(1, 3), "lmin": length, "lmax": length,
                    "dmin": d, "dmax": d}
        return {"kind": kind, "mode": mode, "n": _log_uniform(rng, 16, 2048), "lmin": _log_uniform(rng, 50, 500),
                "lmax": _log_uniform(rng, 1000, 10000), "dmin": 0.005, "dmax": rng.uniform(0.01, 0.05)}
    if kind == "selector":
        lmin = _log_uniform(rng, 50, 5000)
        return {"kind": kind, "n": _log_uniform(rng, 1, 512), "lmin": lmin, "lmax": _log_uniform(rng, lmin, 20000)}
    return {"kind": kind, "n": _log_uniform(rng, 16, 512), "lmax": _log_uniform(rng, 4000, 40000)}


# ---- results -----------------------------------------------------------------------------
# A program keeps the alignments of a submission back to back in buffers that hold any of
# its submissions; what lies past the end of an alignment stays zero.

def _buffers(case):
    kind, n = case["kind"], case.get("n", 1)
    if kind == "serve":
        bases = 8192 * n + 4 * case["lmax"]
        return {"cigars": np.zeros(bases // 2, dtype=np.int32), "ops": np.zeros(bases, dtype=np.uint8)}
    bases = sum(_target_lengths(case))
    if kind == "certified":
        return {k: np.zeros(2 * bases, dtype=np.uint8) for k in ("rows_q", "rows_d", "best_q", "best_d")}
    if kind == "wfa":
        return {"ops": np.zeros(2 * bases + 64, dtype=np.uint8)}
    if kind == "selector":
        return {"hashes": np.zeros(8 * bases, dtype=np.int64), "positions": np.zeros(8 * bases, dtype=np.int32)}
    return {"cigars": np.zeros(bases + 64, dtype=np.int32)}


def _put(buffer, parts):
    """The parts (bytes of the buffer's type) back to back at the start of the buffer."""
    got = np.frombuffer(b"".join(parts), dtype=buffer.dtype)
    buffer[:len(got)] = got
    return buffer


# ---- inputs ------------------------------------------------------------------------------

def _target_lengths(case):
    """Target lengths of a case: spread evenly over their logarithm, the same for every seed."""
    n = case.get("n", 1)
    ratio = case["lmax"] / case["lmin"]
    return [int(round(case["lmin"] * ratio ** ((i + 0.5) / n))) for i in range(n)]


def _lengths(rng, case):
    """The target lengths in the order of this seed."""
    return rng.permutation(_target_lengths(case)).tolist()


def _pairs(rng, case, dmin, dmax):
    return [W.divergent_pair(rng, length, dmin, dmax, 4.0) for length in _lengths(rng, case)]


def _single_pair(rng, case):
    t = W.random_dna(rng, case["lmin"])
    q = W.mutate(rng, t, 0.05, 0.01, 3.0)
    cut = case["deletion"]
    if cut and len(q) > 2 * cut:
        at = int(rng.integers(len(q) // 100, len(q) - cut - len(q) // 100))
        q = np.concatenate([q[:at], q[at + cut:]])
    return q, t


def _codes_case(rng, case):
    """Query and target code arrays of a KSW2 case, and the bands (None: full matrix)."""
    if case["kind"] == "banded":
        qs, ts, bands = [], [], []
        for length in _lengths(rng, case):
            t = W.random_dna(rng, length)
            # long indels up to a fiftieth of the interval: most paths stay inside the band
            q = W.repeat_query(rng, t, long_indels=(2, 6), long_max=max(1, length // 50),
                               element=max(20, length // 20))
            qs.append(q)
            ts.append(t)
            bands.append(max(1, min(len(q), len(t)) * case["percent"] // 100))
        return qs, ts, bands
    pairs = _pairs(rng, case, 0.01, 0.15)
    if case.get("ambiguous"):
        for q, t in pairs[::7]:
            t[int(rng.integers(0, len(t)))] = 4
            q[int(rng.integers(0, len(q)))] = 4
    return [q for q, _ in pairs], [t for _, t in pairs], None


def _flag(case):
    if case["kind"] == "singletrack":
        return ksw2.KSW_EZ_SINGLETRACK
    return ksw2.KSW_EZ_GENERIC_SC if case.get("ambiguous") else 0


def _ascii_pairs(rng, case, dmin, dmax):
    return [(W.to_ascii(q), W.to_ascii(t)) for q, t in _pairs(rng, case, dmin, dmax)]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    ksw2.set_traceback_budget(TRACEBACK_BUDGET)
    state = {"case": case, "out": _buffers(case)}
    if kind == "single":
        state["pair"] = _single_pair(rng, case)
    elif kind in ("batch", "banded", "singletrack"):
        qs, ts, bands = _codes_case(rng, case)
        state["call"] = ksw2.BatchCall(qs, ts, MAT, *GAPS, w=bands, flag=_flag(case))
    elif kind == "certified":
        state["pairs"] = [(q.decode(), t.decode()) for q, t in _ascii_pairs(rng, case, 0.005, 0.06)]
    elif kind == "wfa":
        singletrack, mode = _MODES[case["mode"]]
        pairs = _ascii_pairs(rng, case, case["dmin"], case["dmax"])
        state["aligner"] = wfa.WfaAligner(*WFA_PENALTIES, singletrack=singletrack, max_memory_abort=WFA_POOL,
                                          memory_mode=mode)
        state["texts"], state["patterns"] = [q for q, _ in pairs], [t for _, t in pairs]
    elif kind == "selector":
        pairs = _ascii_pairs(rng, case, 0.01, 0.15)
        state["queries"], state["references"] = [q for q, _ in pairs], [t for _, t in pairs]
    else:
        state["requests"] = W.serving_trace(case["n"], seed=seed, lmax=case["lmax"])
        state["server"] = serve.AlignmentServer(MAT, *GAPS, wfa_penalties=WFA_PENALTIES, slots=2, max_batch=1024,
                                                hbm_budget=SERVER_BUDGET)
        state["next_id"] = 0
    return state


# ---- one pass ------------------------------------------------------------------------------

_EZ_WORDS = ctypes.sizeof(ksw2.KswExtz) // 4
_EZ_FIELDS = [0, 1, 2, 3, 4, 5, 6, 7, 9, 10, 11]  # every field but m_cigar and the pointer


def _batch_results(call, out):
    """The ksw_extz_t fields of every pair and the CIGAR words back to back."""
    fields = np.frombuffer(call.ez, dtype=np.int32).reshape(call.n, _EZ_WORDS)[:, _EZ_FIELDS]
    words = [ctypes.string_at(z.cigar, 4 * z.n_cigar) for z in call.ez if z.n_cigar > 0]
    return {"fields": fields, "cigars": _put(out["cigars"], words)}


def run(state):
    kind, out = state["case"]["kind"], state["out"]
    if kind == "single":
        r = ksw2.ksw_extd2(*state["pair"], MAT, *GAPS)
        out["cigars"][:r.n_cigar] = r.cigar
        return {"fields": np.array(r.key()[:-1], dtype=np.int64), "cigars": out["cigars"]}
    if kind in ("batch", "banded", "singletrack"):
        state["call"].run()
        return _batch_results(state["call"], out)
    if kind == "certified":
        case = state["case"]
        res = ksw2.align_score_certified_ksw2_batch(state["pairs"], case["band"], case["band_max"],
                                                    *ANCHORWAVE_PENALTIES)
        return {"scores": np.array([(r.status == ksw2.CERT_COMPLETED, r.score, r.optimal_score, r.final_band_width,
                                     r.traceback_attempts) for r in res], dtype=np.int64),
                "rows_q": _put(out["rows_q"], [r.alignment_q.encode() for r in res]),
                "rows_d": _put(out["rows_d"], [r.alignment_d.encode() for r in res]),
                "best_q": _put(out["best_q"], [r.best_effort_query_alignment.encode() for r in res]),
                "best_d": _put(out["best_d"], [r.best_effort_reference_alignment.encode() for r in res])}
    if kind == "wfa":
        res, _ = state["aligner"].align_batch(state["patterns"], state["texts"])
        return {"scores": np.array([r[:2] for r in res], dtype=np.int64),
                "ops": _put(out["ops"], [r[2].encode() for r in res])}
    if kind == "selector":
        got, identical, hashes, positions, _ = selector.sequence_summary_raw(state["queries"], state["references"],
                                                                             copy=False)
        out["hashes"][:len(hashes)] = hashes.view(np.int64)
        out["positions"][:len(positions)] = positions.view(np.int32)
        # aw_sequence_summary_t: fingerprint, three fractions, three offsets, three counts
        words = np.frombuffer(got, dtype=np.int64).reshape(2 * len(state["queries"]), 10)
        return {"counts": words[:, [0, 4, 5, 6, 7, 8, 9]], "fractions": words[:, 1:4].copy().view(np.float64),
                "identical": identical, "hashes": out["hashes"], "positions": out["positions"]}
    server, first, reqs = state["server"], state["next_id"], state["requests"]
    for r in reqs:
        server.submit(first + r.id, r.method, r.query, r.target, band=r.band)
    state["next_id"] = first + len(reqs)
    got = []
    while len(got) < len(reqs):
        got += server.poll(1024, wait_ms=1000)
    rows = [(g.id - first, g.method, g.status) + (g.ksw[:-1] if g.ksw else g.wfa[:2] + (0,) * 10) for g in got]
    return {"results": np.array(rows, dtype=np.int64),
            "cigars": _put(out["cigars"], [np.array(g.ksw[-1], dtype=np.int32).tobytes() for g in got if g.ksw]),
            "ops": _put(out["ops"], [g.wfa[2].encode() for g in got if g.wfa])}


# ---- what a pass cannot do without ---------------------------------------------------------

CELL_OPS = 47        # integer operations of a KSW2 cell with its state byte
SCORE_CELL_OPS = 31  # score only
OFFSET_OPS = 40      # integer operations of one wavefront diagonal (five components and a comparison)


def _mean(case, power):
    """Mean of length**power over the target lengths of a case."""
    lengths = _target_lengths(case)
    return sum(float(x) ** power for x in lengths) / len(lengths)


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    if kind == "serve":
        # lengths log-normal around 2 kb, most of the cells in the full KSW2 requests
        return {"bytes": float(n) * 3300 * 4, "flops": float(n) * 0.75 * 2.4e7 * CELL_OPS}
    one, two = _mean(case, 1), _mean(case, 2)
    seqs = 2.0 * n * one               # a byte per base, read once
    if kind == "single":
        return {"bytes": seqs + one / 2, "flops": two * CELL_OPS}
    if kind in ("batch", "singletrack"):
        return {"bytes": seqs + n * one / 2, "flops": n * two * CELL_OPS}
    if kind == "banded":
        return {"bytes": seqs + n * one / 2, "flops": n * two * 2 * case["percent"] / 100 * CELL_OPS}
    if kind == "certified":
        return {"bytes": seqs + 2 * seqs, "flops": n * two * SCORE_CELL_OPS}
    if kind == "wfa":
        # score about 4.6 per edit, wavefronts as wide as the score allows on average
        d = (case["dmin"] + case["dmax"]) / 2
        return {"bytes": 2 * seqs, "flops": n * (4.6 * d) ** 2 * two / 2 * OFFSET_OPS + seqs}
    # selector: bases in, about one sketch entry of 12 bytes for each base of short sequences
    return {"bytes": seqs + 12.0 * 2 * n * min(3 * one, 6144.0), "flops": seqs * 60}


# ---- 64-bit values -------------------------------------------------------------------------

def exact(case, seed):
    """The selector's three fractions in 64 bits; every other output is a whole number."""
    if case["kind"] != "selector":
        return None
    pairs = _ascii_pairs(np.random.default_rng(seed), case, 0.01, 0.15)
    rows = []
    for seq in (s for pair in pairs for s in pair):
        codes = W.to_codes(seq).astype(np.int64)
        n = len(codes)
        known = codes < 4
        # run length of each known base, then the share of bases in runs of four or more
        starts = np.ones(n, dtype=bool)
        starts[1:] = (codes[1:] != codes[:-1]) | ~known[1:]
        at = np.arange(n)
        run = at - np.maximum.accumulate(np.where(starts, at, 0)) + 1
        low = np.count_nonzero(known & (run >= 4)) / n
        # entropy of each 64-base block over its known bases, weighted by them
        blocks = (n + 63) // 64
        count = np.zeros((blocks, 5))
        np.add.at(count, (at // 64, codes), 1.0)
        valid = count[:, :4].sum(axis=1)
        p = count[:, :4] / np.maximum(valid, 1.0)[:, None]
        entropy = -(p * np.log2(np.where(p > 0, p, 1.0))).sum(axis=1)
        rows.append((np.count_nonzero(~known) / n, float((entropy / 2.0 * valid).sum()) / n, low))
    return {"counts": None, "fractions": np.array(rows, dtype=np.float64), "identical": None, "hashes": None,
            "positions": None}
