"""Window consensus against the oracle (byte-identical) where only part of the
graph is a layer's, where sinks tie, and where full CTAs of one-warp teams
share the queue: partial layers in rows of one and of several passes, int16 and
int32 rows, wide alphabets with aligned groups of more than 32 nodes; ends of
layers that leave many tied sinks in groups without a backbone node."""
import random

import pytest

pytestmark = pytest.mark.gpu

WIDE = "".join(map(chr, range(48, 48 + 44)))


def _noisy(rng, s, err, letters):
    out = []
    for c in s:
        u = rng.random()
        if u < err / 3:
            continue
        out.append(rng.choice(letters) if u < 2 * err / 3 else c)
        if rng.random() < err / 3:
            out.append(rng.choice(letters))
    return "".join(out) or rng.choice(letters)


def _window(rng, length, n, letters, err, partial=0.6, tail=0):
    truth = "".join(rng.choice(letters) for _ in range(length))
    w = {"backbone": truth, "backbone_quality": None, "layers": [], "qualities": [], "begins": [], "ends": [],
         "tgs": rng.randrange(2)}
    for k in range(n):
        b, e = 0, length - 1
        if rng.random() < partial and length > 4:
            b = rng.randrange(0, length // 2)
            e = rng.randrange(b + 1, length)
        s = _noisy(rng, truth[b:e + 1], err, letters)
        if tail:
            # bases past the backbone's end: sinks that only layers have
            s += "".join(rng.choice(letters) for _ in range(rng.randrange(tail + 1)))
        w["layers"].append(s)
        w["qualities"].append("".join(chr(33 + rng.randint(0, 40)) for _ in s) if k % 2 else None)
        w["begins"].append(b)
        w["ends"].append(e)
    return w


def _check(native_lib, oracle_lib, wins, m, x, g, forms=(False, True)):
    want = [oracle_lib.window_consensus(w, m, x, g, True)[:2] for w in wins]
    with native_lib.Context(0, m, x, g, 500) as ctx:
        ctx.poa_stage(wins)
        for plain in forms:
            ctx.poa_run(plain=plain)
            got = ctx.poa_fetch()
            bad = [i for i in range(len(wins)) if got[i] != want[i]]
            assert not bad, "plain=%s: windows %s differ" % (plain, bad[:10])


@pytest.mark.parametrize("letters,m,x,g", [("ACGT", 3, -5, -4), ("ACGT", 5, -4, -8), ("ACGT", 20, -20, -30),
                                           ("ACGTN", 1, -1, -1), (WIDE, 3, -5, -4)])
@pytest.mark.parametrize("length", [40, 500, 800, 1100, 1700])
def test_partial_layers(native_lib, oracle_lib, length, letters, m, x, g):
    rng = random.Random(length * 7 + m + len(letters))
    wins = [_window(rng, length, 9, letters, 0.15) for _ in range(3)]
    _check(native_lib, oracle_lib, wins, m, x, g)


@pytest.mark.parametrize("length", [60, 300])
def test_groups_of_more_than_32_nodes(native_lib, oracle_lib, length):
    # substitutions only, every other letter of the alphabet at every place
    rng = random.Random(length)
    wins = []
    for _ in range(2):
        w = _window(rng, length, 0, WIDE, 0)
        for k in range(60):
            b, e = (0, length - 1) if k % 3 else (rng.randrange(length // 2), rng.randrange(length // 2 + 1, length))
            s = "".join(c if rng.random() < 0.3 else rng.choice(WIDE) for c in w["backbone"][b:e + 1])
            w["layers"].append(s)
            w["qualities"].append(None)
            w["begins"].append(b)
            w["ends"].append(e)
        wins.append(w)
    _check(native_lib, oracle_lib, wins, 1, 0, -20)
    _check(native_lib, oracle_lib, wins, 3, -1, -4)


# tails up to 8 bases: groups at the graph's end; up to 1100: past the rows that
# are swept for their order
@pytest.mark.parametrize("m,x,g", [(0, 0, 0), (1, 1, 0), (1, 0, 0), (1, -1, -1), (3, -5, -4)])
@pytest.mark.parametrize("tail", [3, 8, 1100])
def test_tied_ends(native_lib, oracle_lib, tail, m, x, g):
    rng = random.Random(tail + 31 * m + g)
    wins = [_window(rng, rng.randrange(*((20, 120) if tail < 100 else (100, 160))), rng.randrange(4, 16), rng.choice(["AC", "ACGT", WIDE]), 0.2,
                    partial=0.3, tail=tail) for _ in range(24 if tail < 100 else 4)]
    _check(native_lib, oracle_lib, wins, m, x, g)


@pytest.mark.parametrize("letters", ["ACGT", WIDE])
def test_full_ctas_of_one_warp_teams(native_lib, oracle_lib, letters):
    # more windows than four per SM: one warp each, four teams to a CTA
    rng = random.Random(len(letters))
    wins = [_window(rng, rng.randrange(30, 90), rng.randrange(2, 9), letters, 0.15) for _ in range(900)]
    _check(native_lib, oracle_lib, wins, 3, -5, -4, forms=(False,))
