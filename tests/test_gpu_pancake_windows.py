"""Top-down pancake levels in windows of 8! states against the general
path (windows of 2^16 states, asked for by window_bits): the same counts,
children and final arrays, for every algorithm, block shape and far-mark mode,
with flagged (sparse) and full levels and levels that stop part-way."""
import pytest

import puzzlesearch_b200 as psb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,max_depth", [(11, 0), (11, 5), (11, 9), (12, 8)])
@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "classic"])
def test_equal_to_general_path(n, max_depth, algo):
    p = psb.PancakeSimple(n)
    start = p.IndexesCount() * 5 // 7
    want = psb.bfs(p, algo, start, max_depth=max_depth, window_bits=16, direction="top_down", final=True, levels=True)
    variants = [{}] + ([{"threads": 128}, {"threads": 512}] if algo != "classic" else [])
    if algo == "two_bit":
        variants += [{"far_marks": m} for m in ("none", "all")]
    for kw in variants:
        got = psb.bfs(p, algo, start, max_depth=max_depth, direction="top_down", final=True, levels=True, **kw)
        for key in ("counts", "final", "level_children"):
            assert got[key] == want[key], (kw, key)


@pytest.mark.parametrize("n", [11, 12])
def test_mixed_directions(n):
    """Bottom-up levels read and leave the flags that these levels use."""
    p = psb.PancakeSimple(n)
    for algo in ("two_bit", "three_bit", "classic"):
        want = psb.bfs(p, algo, 3, window_bits=16)["counts"]
        assert psb.bfs(p, algo, 3)["counts"] == want
        assert psb.bfs(p, algo, 3, bottom_up_ratio=3.0)["counts"] == want
