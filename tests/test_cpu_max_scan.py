"""The running maximum over a warp's lanes in the consensus DP's rows
(racon_b200/csrc/poa_consensus.cu, dp_strip), restated in Python: shuffles by 1
to 3 lanes, then by 4, 8 and 12, then by 16, a lane that a shuffle does not
reach keeping its own value. It must equal the exact prefix maximum."""
import random


def shuffle_up(x, d):
    return [x[l] if l < d else x[l - d] for l in range(32)]


def scan(x):
    for shifts in ((1, 2, 3), (4, 8, 12), (16,)):
        moved = [shuffle_up(x, d) for d in shifts]
        x = [max([x[l]] + [m[l] for m in moved]) for l in range(32)]
    return x


def test_scan_by_fours_is_the_prefix_maximum():
    rng = random.Random(4)
    for it in range(3000):
        spread = rng.choice([1, 10, 1 << 29])
        x = [rng.randint(-spread, spread) for _ in range(32)]
        if it % 3 == 0:  # one lane decides all that follow
            x[rng.randrange(32)] = 1 << 30
        assert scan(x) == [max(x[:l + 1]) for l in range(32)]
