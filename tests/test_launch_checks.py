"""Arguments that a launcher refuses before anything runs: plain integers stand for device pointers here, so no GPU is needed
(and where one is there, nothing is launched)."""
import pytest

from omegalax_b200.ops import lib

A = 1 << 20      # an aligned address that is never read


@pytest.mark.parametrize("h,out,D,code", [(A + 2, A, 64, 6002), (A, A + 8, 64, 6002), (A, A, 60, 6001)])
def test_row_gather_of_the_head_wants_16_byte_rows(h, out, D, code):
    """A contiguous view may start anywhere; the gather reads 16 bytes at a time, as the products it stands before do."""
    assert lib.load().ob_ce_gather(h, A, A, out, 128, D, None) == code
