"""The work a user of this framework has it do, as measurable cases.

listed() covers the three things a program calls the framework for:

  consensus  window consensus: a batch of windows (backbone + layers) to their
             consensus bytes, staged once and run (Context.poa_stage, then
             poa_run + poa_fetch), or from host strings in one call
             (Context.poa, "host": True);
  align      overlap alignment: query/target spans to edit distances, breaking
             points and optionally CIGARs (Context.align_prepared);
  polish     a whole job, files in and FASTA out (polish_files), contig
             polishing or read correction ("fragment": True);
  serve      several jobs at once through the serving loop (Server).

Shapes follow the repository's own configurations: -w 500 (and 200, 1000),
scores 3/-5/-4, 5/-4/-8 and 1/-1/-1, depth up to 200, 8-15% read error, reads
with and without qualities, overlaps of 1-50 kb and longer.
"""
import ctypes
import math
import os
import tempfile

import numpy as np

import racon_b200
from racon_b200 import synthetic

_BASES = np.frombuffer(b"ACGT", dtype=np.uint8)


def listed():
    return [
        # one short-coverage window, the smallest call: launch and chain latency
        dict(name="window_one", kind="consensus", host=True, windows=1, window_length=500, depth=12, error=0.12,
             quality=False, match=3, mismatch=-5, gap=-4, trim=True),
        # a 20 kb serving job: few windows, the GPU is far from full
        dict(name="windows_small_job", kind="consensus", host=False, windows=40, window_length=500, depth=24,
             error=0.08, quality=False, match=3, mismatch=-5, gap=-4, trim=True),
        # 1 Mb at 50x FASTQ, the benchmark's batch
        dict(name="windows_1mb_50x", kind="consensus", host=False, windows=2001, window_length=500, depth=50,
             error=0.12, quality=True, match=3, mismatch=-5, gap=-4, trim=True),
        # -w 1000 with the reference tests' scores: rows over 768 columns
        dict(name="windows_w1000", kind="consensus", host=False, windows=150, window_length=1000, depth=20,
             error=0.11, quality=True, match=5, mismatch=-4, gap=-8, trim=True),
        # the deep end of read correction
        dict(name="windows_deep", kind="consensus", host=False, windows=96, window_length=500, depth=120, error=0.15,
             quality=True, match=1, mismatch=-1, gap=-1, trim=False),
        # many short windows (-w 200)
        dict(name="windows_w200", kind="consensus", host=False, windows=4003, window_length=200, depth=20,
             error=0.10, quality=False, match=3, mismatch=-5, gap=-4, trim=True),
        # one overlap, the smallest alignment call
        dict(name="align_one", kind="align", pairs=1, shortest=3000, longest=3000, error=0.15, cigar=True,
             window_length=500),
        # an alignment batch of the benchmark's shape
        dict(name="align_batch", kind="align", pairs=700, shortest=1000, longest=50000, error=0.15, cigar=True,
             window_length=500),
        # a few ultra-long overlaps
        dict(name="align_long", kind="align", pairs=9, shortest=60000, longest=120000, error=0.10, cigar=False,
             window_length=500),
        # a small contig job end to end: 50 kb at 30x, FASTA reads
        dict(name="polish_50kb_30x", kind="polish", fragment=False, genome=50000, coverage=30, mean=5000, error=0.13,
             quality=False, window_length=500, match=3, mismatch=-5, gap=-4),
        # read correction end to end
        dict(name="correct_reads", kind="polish", fragment=True, genome=24000, coverage=30, mean=4000, error=0.15,
             quality=True, window_length=500, match=1, mismatch=-1, gap=-1),
        # four jobs in flight on the serving loop
        dict(name="serve_4_jobs", kind="serve", jobs=4, shortest=20000, longest=90000, coverage=30, error=0.12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["consensus", "consensus", "consensus", "align", "align", "polish"])
    match, mismatch, gap = rng.choice([(3, -5, -4), (5, -4, -8), (1, -1, -1)])
    error = round(rng.uniform(0.08, 0.15), 3)
    if kind == "consensus":
        w = rng.choice([200, 500, 500, 1000, _log_int(rng, 150, 1100)])
        depth = _log_int(rng, 6, 40 if w > 700 else 120)
        # bounded so that a drawn batch costs no more than the largest listed one
        most = min(4003, int(2001 * (50 / depth) ** 1.7 * (500 / w) ** 2))
        if w > 767 or depth > 60:
            most = min(most, 150)
        n = _log_int(rng, 1, max(1, most))
        return dict(kind=kind, host=n < 8, windows=n, window_length=w, depth=depth, error=error,
                    quality=rng.random() < 0.5, match=match, mismatch=mismatch, gap=gap, trim=rng.random() < 0.7)
    if kind == "align":
        longest = _log_int(rng, 500, 120000)
        n = _log_int(rng, 1, max(1, min(700, int(700 * (30000 / longest) ** 1.5))))
        return dict(kind=kind, pairs=n, shortest=max(1, longest // rng.choice([1, 2, 10, 50])), longest=longest,
                    error=error, cigar=rng.random() < 0.5, window_length=rng.choice([200, 500, 1000]))
    fragment = rng.random() < 0.4
    genome = _log_int(rng, 5000, 24000 if fragment else 120000)
    return dict(kind=kind, fragment=fragment, genome=genome, coverage=rng.randint(12, 30 if fragment else 50),
                mean=rng.randint(2000, 4000 if fragment else 8000), error=error, quality=rng.random() < 0.5,
                window_length=500, match=match, mismatch=mismatch, gap=gap)


def _mutated(rng, seq, error):
    """A read of seq (codes 0..3) with the given error, 6:3:3 over
    substitutions, insertions and deletions. Returns the codes and the number
    of read bases before each base of seq (len(seq) + 1 entries)."""
    n = len(seq)
    u = rng.integers(0, 65536, n, dtype=np.uint16)
    quarter = int(error * 65536 / 4)
    dele = u < quarter
    ins = (u >= quarter) & (u < 2 * quarter)
    sub = (u >= 2 * quarter) & (u < 4 * quarter)
    base = seq.copy()
    base[sub] = (seq[sub] + rng.integers(1, 4, int(sub.sum()), dtype=np.uint8)) & 3
    count = np.ones(n, dtype=np.uint8)
    count[dele] = 0
    count[ins] = 2
    at = np.zeros(n + 1, dtype=np.int32)
    np.cumsum(count, dtype=np.int32, out=at[1:])
    out = np.repeat(base, count)
    second = at[1:][ins] - 1
    out[second] = rng.integers(0, 4, len(second), dtype=np.uint8)
    return out, at


def _windows(case, rng):
    """Windows as racon cuts them: a draft's consecutive slices, and per window
    the slices of the reads that cover it. Depth varies from window to
    window; reads start or end inside a window in one layer of eight."""
    n, w = case["windows"], case["window_length"]
    truth = rng.integers(0, 4, n * w, dtype=np.uint8)
    # the last window of a contig is shorter than the others
    length = n * w - int(rng.integers(0, w // 2)) if n > 1 else w
    truth = truth[:length]
    cuts = np.minimum(np.arange(n + 1) * w, length)
    draft, at = _mutated(rng, truth, 0.01)
    bounds = at[cuts]
    draft = _BASES[draft].tobytes()
    windows = []
    for i in range(n):
        windows.append({"backbone": draft[bounds[i]:bounds[i + 1]], "layers": [], "begins": [], "ends": [],
                        "qualities": [], "tgs": 1, "id": 0, "rank": i})
    depths = np.maximum(3, np.round(rng.normal(case["depth"], 0.13 * case["depth"], n))).astype(np.int64)
    dmap = at
    for d in range(int(depths.max())):
        read, at = _mutated(rng, truth, case["error"])
        qual = (rng.integers(5, 31, len(read), dtype=np.uint8) + 33).tobytes() if case["quality"] else None
        read = _BASES[read].tobytes()
        part = rng.random(n) < 0.125
        frac = rng.random(n) * 0.8 + 0.1
        left = rng.random(n) < 0.5
        for i in np.flatnonzero(depths > d):
            a, b = cuts[i], cuts[i + 1]
            if part[i]:
                c = a + int(frac[i] * (b - a))
                a, b = (c, b) if left[i] else (a, c)
            s, e = int(at[a]), int(at[b])
            lo, hi = int(dmap[a] - bounds[i]), int(dmap[b] - bounds[i]) - 1
            if e - s < max(2, 0.02 * w) or lo >= hi:
                continue
            x = windows[i]
            x["layers"].append(read[s:e])
            x["qualities"].append(qual[s:e] if qual is not None else None)
            x["begins"].append(lo)
            x["ends"].append(hi)
    return windows


class _State:
    pass


def _files(case, seed, folder):
    if case["fragment"]:
        r, o, t, _ = synthetic.fragment(folder, genome=case["genome"], contigs=1,
                                        depth=(case["coverage"] // 3, case["coverage"]), mean=case["mean"],
                                        sd=case["mean"] // 3, err=case["error"], seed=seed)
        return r, o, t
    e = case["error"]
    shape = dict(genome=case["genome"], coverage=case["coverage"], mean=case["mean"], sd=case["mean"] // 2, lo=500,
                 hi=50000, read_err=(e * 5 / 13, e * 4 / 13, e * 4 / 13), fastq=case["quality"],
                 jitter=50 if case["quality"] else 0)
    r, o, t, _ = synthetic.contig(folder, 0, seed=seed, params=shape)
    return r, o, t


_server = None


def _the_server():
    """One serving loop per program, as a service keeps it."""
    global _server
    if _server is None:
        _server = racon_b200.Server(0, workers=4, hbm_budget=60 << 30)
    return _server


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = _State()
    s.case = case
    s.out = np.zeros(_room(case), dtype=np.uint8)
    if case["kind"] == "consensus":
        s.ctx = racon_b200.Context(0, case["match"], case["mismatch"], case["gap"], case["window_length"])
        s.windows = _windows(case, rng)
        if not case["host"]:
            s.ctx.poa_stage(s.windows, trim=case["trim"])
    elif case["kind"] == "align":
        s.ctx = racon_b200.Context(0, window_length=case["window_length"])
        e = case["error"]
        pairs = synthetic.pairs(case["pairs"], case["shortest"], case["longest"], seed=seed,
                                err=(e * 7 / 15, e * 4 / 15, e * 4 / 15))
        s.pairs = s.ctx.prepare_pairs(pairs)
        s.points = np.zeros(4 * case["pairs"] * (case["longest"] // case["window_length"] + 2), dtype=np.uint32)
    elif case["kind"] == "polish":
        s.folder = tempfile.TemporaryDirectory(prefix="polish_")
        s.files = _files(case, seed, s.folder.name)
    else:
        s.folder = tempfile.TemporaryDirectory(prefix="serve_")
        s.server = _the_server()
        s.out = [np.zeros(_room(case), dtype=np.uint8) for _ in range(case["jobs"])]
        s.files = []
        sizes = np.exp(np.linspace(np.log(case["shortest"]), np.log(case["longest"]), case["jobs"]))
        for i, genome in enumerate(sizes):
            job = dict(fragment=False, genome=int(genome), coverage=case["coverage"], mean=5000, error=case["error"],
                       quality=i % 2 == 1)
            s.files.append(_files(job, int(rng.integers(1 << 31)), os.path.join(s.folder.name, "job%d" % i)))
    return s


def _room(case):
    """Values a case's largest output can take: results come in buffers of a
    size that the case alone decides, padded with zeros."""
    if case["kind"] == "consensus":
        return case["windows"] * 2 * (case["window_length"] + 16)
    if case["kind"] == "align":
        # CIGAR text stays below the target's bases at these error rates
        return case["pairs"] * (case["shortest"] + case["longest"]) // 2 + 4 * case["longest"]
    if case["kind"] == "polish":
        return int(case["genome"] * 1.3 * (case["coverage"] if case["fragment"] else 1)) + 4096
    return int(case["longest"] * 1.3) + 4096


def _put(buffer, data):
    n = len(data)
    buffer[:n] = data
    buffer[n:] = 0
    return buffer


def _view(pointer, n, dtype):
    """n values of a library-owned result array."""
    if n == 0:
        return np.zeros(0, dtype=dtype)
    raw = (ctypes.c_char * (int(n) * np.dtype(dtype).itemsize)).from_address(
        ctypes.cast(pointer, ctypes.c_void_p).value)
    return np.frombuffer(raw, dtype=dtype)


def _text(buffer, fasta):
    return _put(buffer, np.frombuffer(fasta.encode(), dtype=np.uint8))


def run(state):
    case = state.case
    if case["kind"] == "consensus":
        if case["host"]:
            results = state.ctx.poa(state.windows, trim=case["trim"])
        else:
            state.ctx.poa_run()
            results = state.ctx.poa_fetch()
        return {"consensus": _text(state.out, "".join(c for c, _ in results)),
                "lengths": np.array([len(c) for c, _ in results], dtype=np.int64),
                "polished": np.array([p for _, p in results], dtype=np.uint8)}
    if case["kind"] == "align":
        n = state.pairs[2]
        r = state.ctx.align_prepared(state.pairs, want_cigar=case["cigar"])
        offsets = _view(r.bp_offsets, n + 1, np.int64)
        out = {"distance": _view(r.edit_distance, n, np.int32).copy(), "offsets": offsets.copy(),
               "breakpoints": _put(state.points, _view(r.breakpoints, offsets[-1], np.uint32))}
        if case["cigar"]:
            offsets = _view(r.cigar_offsets, n + 1, np.int64)
            out["cigar_offsets"] = offsets.copy()
            out["cigars"] = _put(state.out, _view(r.cigars, offsets[-1], np.uint8))
        return out
    if case["kind"] == "polish":
        return _text(state.out, racon_b200.polish_files(*state.files, fragment=case["fragment"],
                                                        window_length=case["window_length"], match=case["match"],
                                                        mismatch=case["mismatch"], gap=case["gap"]))
    tickets = [state.server.submit(*f) for f in state.files]
    return [_text(buffer, state.server.wait(t)[0]) for t, buffer in zip(tickets, state.out)]


def _consensus_work(windows, w, depth, error, quality):
    # a layer is compared with every node of the graph so far; the graph grows
    # with the layers' errors
    nodes = w * (1 + 0.19 * error * depth)
    cells = windows * depth * w * nodes
    data = windows * w * (1 + depth) * (2 if quality else 1)
    # three max-plus operations per cell
    return {"bytes": data + windows * w, "flops": 3 * cells}


def _align_work(pairs, length, error):
    # the band of an alignment within its edit distance, in 64-row bit vectors of about 17 operations a step
    d = max(1.0, error * length)
    return {"bytes": pairs * 2 * length, "flops": pairs * 17 * length * max(1.0, d / 64)}


def work(case):
    if case["kind"] == "consensus":
        return _consensus_work(case["windows"], case["window_length"], case["depth"], case["error"], case["quality"])
    if case["kind"] == "align":
        lengths = np.linspace(case["shortest"], case["longest"], 16)
        parts = [_align_work(case["pairs"] / 16, x, case["error"]) for x in lengths]
    elif case["kind"] == "polish":
        # read correction polishes every read, each covered like the genome
        targets = case["genome"] * (case["coverage"] * 2 / 3 if case["fragment"] else 1)
        depth = case["coverage"] * (2 / 3 if case["fragment"] else 1)
        parts = [_consensus_work(targets / case["window_length"], case["window_length"], depth, case["error"],
                                 case["quality"]),
                 _align_work(targets * depth / case["mean"], case["mean"], case["error"])]
    else:
        sizes = np.exp(np.linspace(np.log(case["shortest"]), np.log(case["longest"]), case["jobs"]))
        parts = []
        for genome in sizes:
            parts.append(_consensus_work(genome / 500, 500, case["coverage"], case["error"], False))
            parts.append(_align_work(genome * case["coverage"] / 5000, 5000, case["error"]))
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}
