"""Scores whose mismatch is above their match, at layer lengths whose slanted
scores leave 16 bits: the score rows then have to be 32-bit. Against the oracle
(byte-identical), four warps a window (poa_run on a batch this small) and one
(the plain form)."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _noisy(rng, s, err):
    out = []
    for c in s:
        u = rng.random()
        if u < err / 3:
            continue
        out.append(rng.choice("ACGT") if u < 2 * err / 3 else c)
        if rng.random() < err / 3:
            out.append(rng.choice("ACGT"))
    return "".join(out)


@pytest.mark.parametrize("m,x,g,length", [
    (5, 60, -60, 500),
    (-1, 20, -40, 700),
    (0, 100, -1, 500),
    (-128, 100, -27, 300),
    (100, -20, -27, 300),
])
def test_mismatch_above_match(native_lib, oracle_lib, m, x, g, length):
    rng = random.Random(length + x)
    wins = []
    for _ in range(3):
        truth = "".join(rng.choice("ACGT") for _ in range(length))
        layers = [_noisy(rng, truth, 0.15) for _ in range(5)]
        wins.append({"backbone": truth, "backbone_quality": None, "layers": layers, "qualities": [None] * len(layers),
                     "begins": [0] * len(layers), "ends": [length - 1] * len(layers), "tgs": 1})
    want = [oracle_lib.window_consensus(w, m, x, g, True)[:2] for w in wins]
    with native_lib.Context(0, m, x, g, 500) as ctx:
        ctx.poa_stage(wins)
        for plain in (False, True):
            ctx.poa_run(plain=plain)
            assert ctx.poa_fetch() == want, "plain=%s" % plain
