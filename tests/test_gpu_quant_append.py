"""The quantising append over token pairs: sequences that start and end on either side of a pair (needs a B200)."""
import pytest

from kvcase import Pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128, 256])
def test_pages_hold_the_oracles_bytes_whatever_the_parity(d):
    # ragged steps: one token to several pages, from even and odd positions, pairs whose other token is an earlier step's;
    # packed words and scales are compared bit for bit
    p = Pair(1, 8, 2, d, 512, num_pages=100, seed=d, shuffle_free_list=True, quantize_kv=True)
    seqs = [p.new_seq() for _ in range(5)]
    for new in ([1, 2, 3, 16, 33], [2, 1, 1, 3, 15], [17, 16, 5, 1, 2], [1, 40, 31, 2, 4], [3, 3, 3, 3, 3], [2, 100, 1, 64, 7]):
        p.step(seqs, new)
        p.assert_state_equal("used")
    p.step([seqs[3]], [29])
    p.step([seqs[0]], [1])
    p.assert_state_equal("used")
