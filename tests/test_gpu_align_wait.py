"""A wait between the warps that sweep a pair's strips that runs out gives the
pass up with an error status, and the context stays usable. The limit is
shortened to a few polls, less than the strip above takes to its first words;
nothing hangs and nothing faults."""
import random

import pytest

pytestmark = pytest.mark.gpu


# CTAs of four warps, and of eight
@pytest.mark.parametrize("length", [9000, 66000])
def test_expired_wait_is_an_error(native_lib, oracle_lib, monkeypatch, length):
    rng = random.Random(length)
    t = "".join(rng.choice("ACGT") for _ in range(length))
    q = t[:length // 2] + t[length // 2 + 2500:]  # a gap wider than the diagonal form's bands
    pair = [{"query": q, "target": t}]
    with native_lib.Context(0) as ctx:
        monkeypatch.setenv("RB_NW_WAIT_POLLS", "2")
        with pytest.raises(native_lib.RaconB200Error, match="status 6"):
            ctx.align(pair)
        monkeypatch.delenv("RB_NW_WAIT_POLLS")
        got = ctx.align(pair)
        assert (got[0]["edit_distance"], got[0]["cigar"]) == oracle_lib.nw_cigar(q, t)
