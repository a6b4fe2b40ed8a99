"""Searches that run whole in one launch, against the oracle and the
level-by-level path (asked for by window_bits): index spaces from two states
to the largest that run this way, not multiples of a block's share or of 64,
all directions, searches stopped part-way, packed indexes and peg symmetry."""
import pytest

import oracle as O
import puzzlesearch_b200 as psb
from _puzzles import make

pytestmark = pytest.mark.gpu

SPECS = ([["pancake", n, 0] for n in (2, 3, 6, 7, 9)] + [["sliding", w, h] for w, h in ((1, 2), (2, 2), (7, 1), (2, 4), (3, 3))]
         + [["hanoi4", n, s] for n, s in ((1, 0), (2, 1), (5, 0), (8, 1), (9, 0))]
         + [["sliding_opt", 2, 2], ["sliding_opt", 3, 3], ["hanoi4_opt", 8, 1], ["pancake_opt", 8, 0]])


@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "classic"])
@pytest.mark.parametrize("spec", SPECS, ids=lambda s: f"{s[0]}{s[1]}x{s[2]}")
def test_counts_and_final_arrays(spec, algo):
    p = make(spec)
    n = p.IndexesCount()
    if spec[0] == "sliding_opt":
        starts = [O.parse(spec, " ".join(str(i) for i in range(spec[1] * spec[2])))]
    else:
        starts = {0, n - 1, n * 5 // 7} if not spec[2] or spec[0] == "sliding" else {0}
    for start in starts:
        counts, final = O.bfs(spec, algo, start, final=True)
        for direction in ("auto", "top_down", "bottom_up"):
            r = psb.bfs(p, algo, start, final=True, direction=direction)
            if direction != "bottom_up" or spec[2] == 1 or n <= 1 << 17:  # larger bottom-up searches go level by level
                assert r["stats"]["expand_launches"] == 1
            assert r["counts"] == counts and r["final"] == final, direction
        for md in {1, 2, len(counts) // 2, len(counts) - 1, len(counts) + 3} - {0}:
            r = psb.bfs(p, algo, start, final=True, max_depth=md)
            want = psb.bfs(p, algo, start, final=True, max_depth=md, window_bits=10)
            assert want["stats"]["expand_launches"] > 1 or len(counts) == 1 or md < 2
            assert r["counts"] == counts[:md + 1]
            assert r["final"] == want["final"], md


@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "classic"])
@pytest.mark.parametrize("disks", [10, 11])
def test_largest_hanoi(disks, algo):
    """The largest Hanoi searches that run this way, against the level-by-level path."""
    p = psb.FourPegHanoiSimple(disks)
    for start in (0, p.IndexesCount() * 5 // 7):
        r = psb.bfs(p, algo, start, final=True)
        want = psb.bfs(p, algo, start, final=True, window_bits=12)
        assert r["stats"]["expand_launches"] == 1 < want["stats"]["expand_launches"]
        assert r["counts"] == want["counts"] and r["final"] == want["final"]


def test_children_and_sessions():
    """Children per depth without level times; a session's arrays hold no
    trace of the search before."""
    p = psb.SlidingTilePuzzleSimple(3, 3)
    want = psb.bfs(p, "two_bit", 5, direction="top_down", window_bits=10)["stats"]
    got = psb.bfs(p, "two_bit", 5, direction="top_down")["stats"]
    assert (got["children"], got["expanded"], got["levels"]) == (want["children"], want["expanded"], want["levels"])
    s = psb.BfsSession(p, "two_bit")
    for start in (5, 0, 5, 362879):
        assert s.run(start)[0] == O.bfs(["sliding", 3, 3], "two_bit", start)[0]
    s.close()
