"""Hanoi levels taken 64 states at a time, against the oracle: the smallest
searches that run them (three disks: one unit), searches of one window and of
many (moves inside and across windows), every algorithm, block shape and
far-mark mode, from starts with empty pegs and from random ones."""
import pytest

import oracle as O
import puzzlesearch_b200 as psb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "classic", "frontier"])
@pytest.mark.parametrize("disks,window_bits", [(2, 10), (3, 10), (4, 10), (5, 12), (6, 10), (7, 11), (8, 10), (9, 16)])
def test_final_arrays(algo, disks, window_bits):
    p = psb.FourPegHanoiSimple(disks)
    n = p.IndexesCount()
    for start in {0, n - 1, (0x2D2D2D2D2D & (n - 1)), 0x123456789 % n}:
        counts, final = O.bfs(["hanoi4", disks, 0], algo, start, final=True)
        for kw in [{}] + ([{"threads": 128}, {"threads": 512}] if algo in ("two_bit", "three_bit") else []) + (
                [{"far_marks": "near"}, {"far_marks": "all", "threads": 128}] if algo == "two_bit" else []):
            r = psb.bfs(p, algo, start, final=True, window_bits=window_bits, direction="top_down", **kw)
            assert r["counts"] == counts, kw
            assert r["final"] == final, kw


def test_children_per_depth():
    """Children generated from each depth equal the oracle's expansions."""
    p = psb.FourPegHanoiSimple(6)
    n = p.IndexesCount()
    for start in (0, 0x9C5):
        depth = O.depths(["hanoi4", 6, 0], start)[0]
        r = psb.bfs(p, "two_bit", start, levels=True, direction="top_down")
        want = [0] * len(r["counts"])
        for i in range(n):
            want[depth[i]] += len(O.expand(["hanoi4", 6, 0], [i])[0])
        assert r["level_children"] == want
