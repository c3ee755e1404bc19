"""The quantising append, by rows and over token pairs: sequences that start and end on either side of a pair (needs a B200)."""
import pytest
import torch

from combsengine_b200 import KVArena
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


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("k_off,v_off", [(4, 0), (0, 4), (4, 12)])
def test_rows_that_start_at_8_bytes_fill_the_same_pages(d, k_off, v_off):
    # contiguous views into larger buffers, as a fused projection leaves them; one call appends, the other attends as well
    gen = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    view = lambda x, off: torch.zeros(x.numel() + 16, dtype=x.dtype, device="cuda")[off:off + x.numel()].copy_(x)
    # (801 tokens of 8 heads: over token pairs at a multiple of 16, a row per warp otherwise)
    g = KVArena(1, 8, 8, d, 1024, 16, 64, quantize_kv=True)
    s = g.new_seq()
    n = 801
    q, k, v = (rand(n * 8 * d) for _ in range(3))

    def pages(kx, vx):
        g.begin_step([s], [n])
        out = g.attention(0, q, kx, vx, d ** -0.5)
        rows = [g.export_page_quant(0, int(page)) for page in s.block_table()]
        s.popn(n)
        return out, rows

    out, rows = pages(k, v)
    out8, rows8 = pages(view(k, k_off), view(v, v_off))
    assert g.device_status() == 0
    assert torch.equal(out, out8)
    assert all((x == y).all() for a, b in zip(rows, rows8) for x, y in zip(a, b))


@pytest.mark.parametrize("d", [64, 128, 256])
def test_large_steps_hold_the_oracles_bytes_whatever_the_parity(d):
    # 12288 rows and more, over token pairs; the last step is just below, a row per warp
    p = Pair(1, 8, 8, d, 2048, num_pages=400, seed=d, shuffle_free_list=True, quantize_kv=True)
    seqs = [p.new_seq() for _ in range(5)]
    for new in ([1, 2, 333, 16, 433], [2, 301, 1, 3, 512], [417, 316, 5, 33, 1], [160, 161, 1, 160, 286], [160, 160, 1, 160, 286]):
        p.step(seqs, new)
        p.assert_state_equal("used")
