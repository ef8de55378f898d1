"""No capture on any board reaches the depth limit of the capture walk (15
jumps): a jump moves two rows and two columns and no square is landed on twice,
so a piece has at most eight landing squares.  Boards on which a king's squares
of that class are free and the squares between them are taken, all of them or
most, for kings of every square and either side: the walk ends, the longest
captures take at least six pieces and none more than eight."""
import numpy as np

from golden_boards import sq
from test_rules_host import rh, rh_genmoves  # noqa: F401  (rh is a fixture)


def _boards():
    rng = np.random.default_rng(3)
    out = []
    dark = [(r, c) for r in range(8) for c in range(8) if (r + c) % 2 == 1]
    for r, c in dark:
        land = {(r2, c2) for r2, c2 in dark if (r2 - r) % 2 == 0 and ((r2 - r) // 2 + (c2 - c) // 2) % 2 == 0}
        assert len(land) == 8
        rest = sum(1 << sq(*s) for s in dark if s not in land)
        for k in range(40):
            opp = rest if k == 0 else rest & ~(int(rng.integers(1 << 32)) & int(rng.integers(1 << 32)))
            own = 1 << sq(r, c)
            turn = k % 2
            out.append([opp if turn else own, own if turn else opp, own | (opp & int(rng.integers(1 << 32))), turn])
    return np.array(out, np.uint32)


def test_no_capture_reaches_the_depth_limit(rh):  # noqa: F811
    longest = 0
    for b in np.array_split(_boards(), 16):
        moves, _ = rh_genmoves(rh, b, 2048)  # fails on a count of -1
        longest = max(longest, int(moves[:, :, 2].max()))
    assert 6 <= longest <= 8
