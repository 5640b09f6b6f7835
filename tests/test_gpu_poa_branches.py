"""Windows whose layers all end inside the window, as short reads do: the best
consensus path then ends at a node with out-edges and is completed branch by
branch. Against the oracle (byte-identical), both team sizes; scores of short
windows sit in shared memory, those of the longest in global memory."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _window(rng, length, n, letters, err):
    truth = "".join(rng.choice(letters) for _ in range(length))
    w = {"backbone": truth, "backbone_quality": None, "layers": [], "qualities": [], "begins": [], "ends": [], "tgs": 0}
    for k in range(n):
        b = rng.randrange(0, length - 1)
        e = rng.randrange(b + 1, min(length, b + 1 + max(2, length // 3)))
        s = "".join(rng.choice(letters) if rng.random() < err else c for c in truth[b:e + 1] if rng.random() > err / 3)
        s = s or "A"
        w["layers"].append(s)
        w["qualities"].append("".join(chr(33 + rng.randint(0, 40)) for _ in s) if k % 2 else None)
        w["begins"].append(b)
        w["ends"].append(e)
    return w


@pytest.mark.parametrize("length,layers,windows", [(12, 3, 40), (60, 8, 40), (500, 12, 12), (500, 60, 4), (3000, 9, 3),
                                                   (6500, 9, 2)])
@pytest.mark.parametrize("letters,m,x,g", [("ACGT", 3, -5, -4), ("AC", 1, -1, -1)])
def test_branch_completion(native_lib, oracle_lib, length, layers, windows, letters, m, x, g):
    rng = random.Random(length + layers + m)
    wins = [_window(rng, length, layers, letters, 0.1) for _ in range(windows)]
    want = [oracle_lib.window_consensus(w, m, x, g, True)[:2] for w in wins]
    with native_lib.Context(0, m, x, g, 500) as ctx:
        ctx.poa_stage(wins)
        for plain in (False, True):
            ctx.poa_run(plain=plain)
            got = ctx.poa_fetch()
            bad = [i for i in range(windows) if got[i] != want[i]]
            assert not bad, "plain=%s: windows %s differ" % (plain, bad)
