"""Layers with more inserted bases before their first matched base than the
starting graph has room for: the window overflows, runs again with four times
the capacity and gives the oracle's consensus (byte-identical); the windows
beside it, whose slots it must not touch, too."""
import random

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("front", [150, 200, 700, 3000])
def test_long_run_before_the_first_anchor(native_lib, oracle_lib, monkeypatch, front):
    rng = random.Random(front)
    truth = "".join(rng.choice("ACG") for _ in range(80))
    plain = truth[:40] + "T" + truth[41:]
    def window(layers):
        return {"backbone": truth, "backbone_quality": None, "layers": layers, "qualities": [None] * len(layers),
                "begins": [0] * len(layers), "ends": [len(truth) - 1] * len(layers), "tgs": 1}
    # no T in the backbone: the layer's front matches nothing and is inserted ahead of it
    long_front = "T" * front + truth
    wins = [window([plain, long_front, truth, plain]), window([plain, truth, plain]), window([long_front, truth, truth, plain])]
    want = [oracle_lib.window_consensus(w, 3, -5, -4, True)[:2] for w in wins]
    monkeypatch.setenv("RB_POA_NCAP", "256")  # 80 nodes and the front: room for 176 new ones
    with native_lib.Context(0, 3, -5, -4, 500) as ctx:
        for run_plain in (False, True):
            ctx.poa_stage(wins)
            ctx.poa_run(plain=run_plain)
            assert ctx.poa_fetch() == want
            assert (ctx.poa_stats().max_nodes > 256) == (front > 176)
