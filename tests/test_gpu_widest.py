"""The widest ranges: windows of 2^19 and 2^20 states (offsets of carried
states take 20 bits; 2^18 with frontier search's operator bits), and frontier
segments of 2^32 states."""
import numpy as np
import pytest

import oracle as O
import puzzlesearch_b200 as psb
from _puzzles import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["two_bit", "three_bit", "classic", "frontier"])
@pytest.mark.parametrize("spec", [["sliding", 2, 5], ["hanoi4", 10, 1], ["hanoi4", 10, 0]],
                         ids=lambda s: f"{s[0]}{s[1]}x{s[2]}")
def test_windows(spec, algo):
    p = make(spec)
    start = 0 if spec[2] == 1 else p.IndexesCount() * 5 // 7
    counts, final = O.bfs(spec, algo, start, final=True)
    for window_bits in (17, 18) if algo == "frontier" else (19, 20):
        r = psb.bfs(p, algo, start, final=True, window_bits=window_bits, direction="top_down")
        assert r["counts"] == counts and r["final"] == final, window_bits


def test_segment_of_all_32_bit_offsets():
    """Thin stretches (StreamVInt) and a dense one up to the last offset (bitmap blocks)."""
    import torch
    rng = np.random.default_rng(32)
    dense = 2**32 - 1 - np.flatnonzero(rng.random(700_000) < 0.8).astype(np.uint64)
    offsets = np.unique(np.concatenate([rng.integers(0, 2**32, 300_000, dtype=np.uint64), dense,
                                        np.array([0, 2**32 - 1], dtype=np.uint64)]))
    words = torch.zeros(1 << 26, dtype=torch.int64, device="cuda")
    at, first = np.unique(offsets >> np.uint64(6), return_index=True)
    value = np.bitwise_or.reduceat(np.uint64(1) << (offsets & np.uint64(63)), first)
    words[torch.from_numpy(at.astype(np.int64)).cuda()] = torch.from_numpy(value.view(np.int64)).cuda()
    want = bytes(O.segment_stream(offsets.astype(np.uint32)))
    out = torch.zeros(len(want) + 64, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    used, blocks, nb = psb.frontier_encode(words.data_ptr(), 0, 2**32, out.data_ptr(), out.numel())
    assert {bool(blocks[i].is_bitmap) for i in range(nb)} == {True, False}
    assert used == len(want) and bytes(out[:used].cpu().numpy()) == want
    back = torch.zeros_like(words)
    torch.cuda.synchronize()
    psb.frontier_decode(out.data_ptr(), blocks, nb, back.data_ptr(), 0, 2**32)
    assert torch.equal(back, words)
