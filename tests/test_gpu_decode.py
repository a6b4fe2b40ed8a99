"""StreamVInt and bitmap blocks decoded tile by tile, against the bitmap they
were encoded from: streams of one tuple to several tiles of 16 KB, deltas of
one to four bytes (chains that never fall into step, and chains that do), all
stream alignments, blocks of both kinds, and streams cut short."""
import numpy as np
import pytest

import oracle as O
import puzzlesearch_b200 as psb

pytestmark = pytest.mark.gpu


def offsets_of(kind, n, rng):
    if kind == "ones":        # every delta 1: five-byte tuples whose chains never meet
        return np.arange(n, dtype=np.uint64)
    if kind == "even":        # one-byte deltas
        return np.cumsum(rng.integers(12, 256, n), dtype=np.uint64)
    if kind == "wide":        # two- and three-byte deltas
        return np.cumsum(rng.integers(200, 70000, n), dtype=np.uint64)
    if kind == "far":         # up to four bytes
        step = max(1, (2**32 - 2) // max(n, 1))
        return np.cumsum(rng.integers(1, step + 1, n), dtype=np.uint64)
    return np.cumsum(rng.choice([1, 3, 255, 256, 65535, 65536], n), dtype=np.uint64)  # descriptors of every form


def decode(data, offsets, n_bits, shift, blocks, nb):
    import torch
    buf = torch.zeros(len(data) + shift, dtype=torch.uint8)
    buf[shift:] = torch.frombuffer(bytearray(data), dtype=torch.uint8)
    d_in = buf.cuda()
    d_bits = torch.zeros((n_bits + 63) // 64, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    psb.frontier_decode(d_in.data_ptr() + shift, blocks, nb, d_bits.data_ptr(), 0, n_bits)
    at = torch.nonzero(d_bits).flatten()
    words = d_bits[at].cpu().numpy().view(np.uint8).reshape(-1, 8)
    w, j = np.nonzero(np.unpackbits(words, axis=1, bitorder="little"))
    assert np.array_equal(at.cpu().numpy()[w] * 64 + j, offsets)


@pytest.mark.parametrize("kind", ["ones", "even", "wide", "far", "mixed"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 100, 129, 5000, 40001])
def test_blocks(kind, n):
    rng = np.random.default_rng(n)
    offsets = offsets_of(kind, n, rng)
    offsets = offsets[offsets < 2**32 - 64]
    if kind == "far" and n > 5000:
        return  # the same range as n = 5000, denser
    n_bits = int(offsets[-1]) + 1
    for encode in (O.svi_encode, O.segment_stream):  # StreamVInt whatever the density; the writer's choice
        data = bytes(encode(offsets.tolist() if encode is O.svi_encode else offsets.astype(np.uint32)))
        blocks, nb = psb.frontier_index(data)
        for shift in ((0, 1, 2, 3) if n in (9, 5000) and kind != "far" else (n % 4,)):
            decode(data, offsets, n_bits, shift, blocks, nb)


def test_many_blocks_and_short_streams():
    rng = np.random.default_rng(5)
    keep = np.concatenate([rng.random(1 << 22) < d for d in (0.4, 0.02, 0.09, 0.3)])
    offsets = np.flatnonzero(keep)
    data = O.segment_stream(offsets.astype(np.uint32))
    blocks, nb = psb.frontier_index(data)
    assert nb > 4 and {bool(blocks[i].is_bitmap) for i in range(nb)} == {True, False}
    decode(data, offsets, len(keep), 1, blocks, nb)
    # a block table that promises more than the bytes it names hold
    for i in range(nb):
        short = (psb.CodecBlock * 1)(psb.CodecBlock(blocks[i].offset, blocks[i].count, blocks[i].bytes - 9,
                                                    blocks[i].first, blocks[i].is_bitmap))
        with pytest.raises(psb.PsbError):
            decode(data, offsets, len(keep), 0, short, 1)
    with pytest.raises(psb.PsbError):  # offsets past the segment
        decode(data, offsets, int(offsets[-1]), 0, blocks, nb)
