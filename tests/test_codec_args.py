"""Arguments that the frontier encoder refuses before it touches the GPU."""
import pytest

import puzzlesearch_b200 as psb


@pytest.mark.parametrize("n_bits", [2**32 + 1, 2**60, 2**64 - 1])
@pytest.mark.parametrize("d_out", [None, 256])
def test_ranges_past_a_segment(n_bits, d_out):
    """Not by running out of host memory for a table of that many blocks."""
    with pytest.raises(psb.PsbError, match="at most 2\\^32 states"):
        psb.frontier_encode(256, 0, n_bits, d_out, 64 if d_out else 0)
