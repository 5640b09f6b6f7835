"""The consensus DP's strips against the oracle (byte-identical) at the sizes
where their shape changes: layer lengths around the widths at which a lane gets
more columns (256, 512, 768, 1024) and rows of several passes; the general form
(int32 rows, characters compared) through other letters and scores that do not
fit the fast one. poa_run takes four warps per window in batches this small,
the plain form one."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _window(rng, length, layers, letters, err=0.1):
    truth = "".join(rng.choice(letters) for _ in range(length))

    def read(n):
        out = []
        for c in truth:
            u = rng.random()
            if u < err / 3:
                continue
            out.append(rng.choice(letters) if u < 2 * err / 3 else c)
            if rng.random() < err / 3:
                out.append(rng.choice(letters))
        out += [rng.choice(letters) for _ in range(max(0, n - len(out)))]
        return "".join(out[:n])

    seqs = [read(length + d) for d in layers]
    return {"backbone": truth, "backbone_quality": None, "layers": seqs,
            "qualities": ["".join(chr(33 + rng.randint(0, 40)) for _ in s) if k % 2 else None
                          for k, s in enumerate(seqs)],
            "begins": [0] * len(seqs), "ends": [length - 1] * len(seqs), "tgs": 1}


def _check(native_lib, oracle_lib, wins, m, x, g):
    want = [oracle_lib.window_consensus(w, m, x, g, True)[:2] for w in wins]
    with native_lib.Context(0, m, x, g, 500) as ctx:
        ctx.poa_stage(wins)
        for plain in (False, True):
            ctx.poa_run(plain=plain)
            got = ctx.poa_fetch()
            bad = [i for i in range(len(wins)) if got[i] != want[i]]
            assert not bad, "plain=%s: windows %s differ" % (plain, bad)


@pytest.mark.parametrize("length", [31, 255, 511, 767, 1023, 1535, 2047])
def test_strip_widths(native_lib, oracle_lib, length):
    rng = random.Random(length)
    wins = [_window(rng, length, (-1, 0, 1, 2, -2), "ACGT") for _ in range(3)]
    _check(native_lib, oracle_lib, wins, 3, -5, -4)


@pytest.mark.parametrize("letters,m,x,g", [
    ("ACGTN", 3, -5, -4),         # another letter: characters compared
    ("ACGTRYKM", 3, -5, -4),      # aligned groups past their inline entries
    ("ACGT", 100, -100, -90),     # s - gap leaves a signed byte
    ("ACGT", 20, -20, -30),       # slanted scores leave 16 bits
    ("ACGT", 3, -5, 0),
])
@pytest.mark.parametrize("length", [200, 520, 1100])
def test_general_form(native_lib, oracle_lib, length, letters, m, x, g):
    rng = random.Random(length + m)
    wins = [_window(rng, length, (0, 3, -3, 1, 5, -1, 2), letters, 0.2) for _ in range(2)]
    _check(native_lib, oracle_lib, wins, m, x, g)


def test_far_and_many_predecessors(native_lib, oracle_lib):
    # deletions of every length up to 60 at one place give a node dozens of
    # in-edges, from rows far above the DP's ring
    rng = random.Random(3)
    truth = "".join(rng.choice("ACGT") for _ in range(300))
    layers = [truth[:100] + truth[100 + k:] for k in range(0, 60)] + [truth] * 3
    win = {"backbone": truth, "backbone_quality": None, "layers": layers, "qualities": [None] * len(layers),
           "begins": [0] * len(layers), "ends": [299] * len(layers), "tgs": 1}
    mirrored = dict(win, backbone=truth[::-1], layers=[s[::-1] for s in layers])
    # more than eight in-edges at one node: sources at every distance
    many = dict(win, layers=[truth[:200 - k] + truth[200:] for k in range(0, 60)] + [truth] * 3)
    _check(native_lib, oracle_lib, [win, mirrored, many], 3, -5, -4)
    _check(native_lib, oracle_lib, [win, mirrored, many], 1, -1, -1)
