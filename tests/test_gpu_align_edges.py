"""Block sweeps at the lengths and bands where their shape changes, against the
oracle: ends of 64-row blocks and 2048-row strips, bands of a single diagonal
(equal sequences, one gap), bands on both sides of the diagonal form's limit,
and alphabets on both sides of its symbol limit."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _mutate(rng, s, err, letters):
    out = []
    for c in s:
        u = rng.random()
        if u < err / 3:
            continue
        out.append(rng.choice(letters) if u < 2 * err / 3 else c)
        if rng.random() < err / 3:
            out.append(rng.choice(letters))
    return "".join(out) or "A"


def _check(native_lib, oracle_lib, pairs):
    with native_lib.Context(0) as ctx:
        got = ctx.align([{"query": q, "target": t} for q, t in pairs])
    for i, ((q, t), g) in enumerate(zip(pairs, got)):
        assert (g["edit_distance"], g["cigar"]) == oracle_lib.nw_cigar(q, t), i


@pytest.mark.parametrize("letters", ["ACGT", "ABCDEFGH", "ABCDEFGHIJKL"])
@pytest.mark.parametrize("length", [1, 63, 64, 65, 2047, 2048, 2049, 4096, 4161])
def test_lengths(native_lib, oracle_lib, length, letters):
    rng = random.Random(length * 31 + len(letters))
    s = "".join(rng.choice(letters) for _ in range(length))
    cut = s[:length // 3] + s[length // 3 + length // 5:] or s
    _check(native_lib, oracle_lib, [(s, s), (cut, s), (s, cut), (_mutate(rng, s, 0.12, letters), s),
                                    (_mutate(rng, s, 0.4, letters), s), (s[::-1], s)])


@pytest.mark.parametrize("shift", [1700, 1899, 1901, 2100, 3900])
def test_bands(native_lib, oracle_lib, shift):
    # one gap of `shift` bases in a noisy overlap: the band's width follows it
    rng = random.Random(shift)
    t = "".join(rng.choice("ACGT") for _ in range(9000))
    q = _mutate(rng, t[:4000] + t[4000 + shift:], 0.05, "ACGT")
    _check(native_lib, oracle_lib, [(q, t), (t, q)])


# Batches of few long pairs are swept by CTAs of four warps (queries from 6144
# bases) and eight (from 65536): both sides of the two lines, strips that wrap
# around the warps and their buffers, passes that give up, wide alphabets.
@pytest.mark.parametrize("length,letters", [(6143, "ACGT"), (6144, "ACGT"), (8193, "ABCDEFGHIJKL"), (10240, "ACGT"),
                                            (10241, "".join(map(chr, range(40, 80)))), (18433, "ACGT"),
                                            (65535, "ACGT"), (65536, "ACGT")])
def test_teams(native_lib, oracle_lib, length, letters):
    rng = random.Random(length)
    s = "".join(rng.choice(letters) for _ in range(length))
    third = s[:length // 3]
    pairs = [(s, third + s[length // 2:]), (_mutate(rng, s, 0.3, letters), s), (s, third)]
    if length < 20000:
        pairs += [(s[::-1], s), (third, s), ("A", s), (_mutate(rng, s, 0.05, letters), s)]
    _check(native_lib, oracle_lib, pairs)
