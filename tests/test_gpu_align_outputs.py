"""Symbol codes, breaking points and CIGARs against the oracle where their work
is shared out differently: pairs taken by one warp (large batches) or by the
eight of a CTA, windows from one base to longer than the target, shares that
begin inside runs, and gaps longer than a lane's and a warp's search."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _pairs(rng, lengths):
    out = []
    for n in lengths:
        t = "".join(rng.choice("ACGT") for _ in range(n))
        kinds = [t,
                 "".join(rng.choice("ACGT") if rng.random() < 0.2 else c for c in t),
                 t[:n // 4] + t[n // 2 + n // 4:] or "A",       # a deletion of half the target
                 t[:n // 2] + "".join(rng.choice("ACGTN") for _ in range(n // 3)) + t[n // 2:],
                 t[n // 2:] or "C", "GT" + t[:n // 3]]
        out += [{"query": q, "target": t, "q_offset": rng.randrange(5000), "t_begin": rng.randrange(5000)}
                for q in kinds]
    return out


@pytest.mark.parametrize("window_length", [1, 7, 33, 64, 500, 1000000])
@pytest.mark.parametrize("large", [False, True])
def test_outputs(native_lib, oracle_lib, window_length, large):
    rng = random.Random(window_length + large)
    lengths = [1, 2, 8, 9, 31, 32, 33, 255, 256, 257, 1000, 2305]
    pairs = _pairs(rng, lengths)
    fill = [{"query": "ACGT", "target": "AGT", "q_offset": 0, "t_begin": 0}] * (2400 if large else 0)
    with native_lib.Context(0, window_length=window_length) as ctx:
        got = ctx.align(pairs + fill)
    for i, (p, g) in enumerate(zip(pairs, got)):
        d, cigar = oracle_lib.nw_cigar(p["query"], p["target"])
        points = oracle_lib.breakpoints(cigar, p["q_offset"], p["q_offset"] + len(p["query"]),
                                        p["q_offset"] + len(p["query"]), p["t_begin"],
                                        p["t_begin"] + len(p["target"]), False, window_length)
        assert (g["edit_distance"], g["cigar"], g["breakpoints"]) == (d, cigar, points), i
    assert all(g == got[len(pairs)] for g in got[len(pairs):])
