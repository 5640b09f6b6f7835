"""A wait between the warps of a window's team that runs out gives the window up
with an error status, and the context stays usable. The limit is shortened to a
few polls, less than the rows take that a warp has to wait for; nothing hangs
and nothing faults."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _windows(rng, length, n):
    out = []
    for _ in range(n):
        truth = "".join(rng.choice("ACGT") for _ in range(length))
        layers = ["".join(c for c in truth if rng.random() > 0.08) for _ in range(5)]
        out.append({"backbone": truth, "backbone_quality": None, "layers": layers, "qualities": [None] * 5,
                    "begins": [0] * 5, "ends": [length - 1] * 5, "tgs": 1})
    return out


# rows of one pass, and of several passes of a four-warp team
@pytest.mark.parametrize("length", [500, 1500])
def test_expired_wait_is_an_error(native_lib, oracle_lib, monkeypatch, length):
    wins = _windows(random.Random(length), length, 3)
    want = [oracle_lib.window_consensus(w, 3, -5, -4, True)[:2] for w in wins]
    with native_lib.Context(0, 3, -5, -4, 500) as ctx:
        ctx.poa_stage(wins)
        monkeypatch.setenv("RB_POA_WAIT_POLLS", "0")
        with pytest.raises(native_lib.RaconB200Error, match="failed on the device"):
            ctx.poa_run()
        monkeypatch.delenv("RB_POA_WAIT_POLLS")
        ctx.poa_run()
        assert ctx.poa_fetch() == want
        # one warp a window waits for no other
        monkeypatch.setenv("RB_POA_WAIT_POLLS", "0")
        ctx.poa_run(plain=True)
        assert ctx.poa_fetch() == want
