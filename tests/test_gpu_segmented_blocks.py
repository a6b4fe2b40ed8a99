"""Segmented searches share a few pinned host blocks: more searches at once
than blocks are kept, blocks given back in between, and searches of so many
segments that they take one of their own."""
import threading

import pytest

import oracle as O
import puzzlesearch_b200 as psb
from _puzzles import make

pytestmark = pytest.mark.gpu

SPECS = [["hanoi4", 6, 0], ["sliding", 2, 4], ["pancake", 7, 0], ["hanoi4", 5, 1], ["sliding", 3, 2], ["pancake", 8, 0]]


def test_searches_at_once():
    want = {tuple(s): O.bfs(s, "three_bit", 0)[0] for s in SPECS}
    wrong = []

    def job(spec):
        p = make(spec)
        for i in range(6):
            counts = psb.bfs_segmented(p, 0, segment_bits=10 + i % 3)["counts"]
            if counts != want[tuple(spec)]:
                wrong.append((spec, counts))

    for _ in range(2):
        threads = [threading.Thread(target=job, args=(s,)) for s in SPECS]
        for t in threads:
            t.start()
        psb.release_cached_memory()
        for t in threads:
            t.join()
        psb.release_cached_memory()
    assert not wrong


def test_many_segments():
    """2^15 segments: their counters do not fit the blocks that are kept."""
    p = make(["hanoi4", 13, 0])
    want = psb.bfs(p, "two_bit", 0, max_depth=6)["counts"]
    for _ in range(2):
        assert psb.bfs_segmented(p, 0, segment_bits=11, max_depth=6)["counts"] == want
