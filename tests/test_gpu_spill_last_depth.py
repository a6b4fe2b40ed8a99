"""A spilled search stopped by max_depth writes its last depth from the
segments that hold some of it; the empty ones cost nothing."""
import pytest

import puzzlesearch_b200 as psb
from _puzzles import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "classic", "frontier"])
@pytest.mark.parametrize("spec", [["hanoi4", 10, 0], ["hanoi4", 10, 1], ["sliding", 2, 5]],
                         ids=lambda s: f"{s[0]}{s[1]}x{s[2]}")
def test_last_depth(spec, algo):
    p = make(spec)
    segments = p.IndexesCount() >> 10  # 1024 and more
    got = {}

    def run(**options):
        got.clear()
        return psb.bfs(p, algo, 0, segment_bits=10, **options,
                       spill=lambda d, g, data, states: got.__setitem__((d, g), (data, states)))

    run(max_depth=8)
    full = dict(got)
    for md in (1, 3, 7):
        r = run(max_depth=md)
        assert got == {k: v for k, v in full.items() if k[0] <= md}
        assert sum(states for _, states in got.values()) == sum(r["counts"])
        assert md > 3 or r["stats"]["spill_launches"] < segments // 2
