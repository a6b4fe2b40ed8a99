"""Depth limits near the end of their 32-bit type: such a search is the
unlimited one, whether it runs whole in one launch or level by level."""
import pytest

import oracle as O
import puzzlesearch_b200 as psb
from _puzzles import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "classic"])
@pytest.mark.parametrize("spec", [["pancake", 7, 0], ["sliding", 3, 3], ["hanoi4", 6, 0], ["hanoi4", 6, 1]],
                         ids=lambda s: f"{s[0]}{s[1]}x{s[2]}")
def test_limit_at_the_end_of_the_type(spec, algo):
    p = make(spec)
    counts, final = O.bfs(spec, algo, 0, final=True)
    for window_bits in (0, 10):
        for md in (2**32 - 1, 2**32 - 2):
            r = psb.bfs(p, algo, 0, final=True, max_depth=md, window_bits=window_bits)
            assert r["counts"] == counts and r["final"] == final, (window_bits, md)
            assert (r["stats"]["expand_launches"] == 1) == (window_bits == 0)
