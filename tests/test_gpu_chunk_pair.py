"""Chunk attention on pairs of SMs, and where the library chooses it, against the oracle (needs a B200)."""
import pytest
import torch

from kvcase import Pair
from test_gpu_chunk_cut import _fill, _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grow", [False, True])
@pytest.mark.parametrize("n_q,n_kv,d", [(28, 4, 128), (32, 8, 128), (8, 8, 128), (8, 4, 256), (8, 1, 256)])
def test_chunks_on_pairs_of_sms(n_q, n_kv, d, grow):
    # tokens per query tile: 16 to 128; chunks that fill one tile, two, and leave the second with none or a few; KV tiles:
    # one, two and many of them, cut and whole
    p = Pair(2, n_q, n_kv, d, 4096, num_pages=1600, windows=[150, None], seed=d + n_q, shuffle_free_list=True, popn_refuses=False,
             chunk_kernel=6)
    for ctx in (0, 1, 50, 130, 900, 2050):
        s = p.new_seq()
        if ctx:
            _fill(p, s, ctx, [0, 1], grow)
    for s in p.seqs:
        _step(p, [s], [70], [0, 1], grow, repeats=5)
        _step(p, [s], [257], [0, 1], grow, repeats=5)
        _step(p, [s], [5 if ctx % 4 else 1], [0, 1], grow, repeats=5)
    _step(p, p.seqs, [128, 65, 80, 129, 200, 97], [0, 1], grow, repeats=20)
    _step(p, p.seqs, [1, 140, 2, 9, 1, 5], [0, 1], grow, repeats=20)
    p.g.set_chunk_split(1)
    _step(p, p.seqs, [128, 65, 80, 129, 200, 97], [0, 1], grow, repeats=5)


def test_prompts_in_both_types_against_64_bits():
    from combsengine_b200 import KVArena
    for dtype in (torch.float16, torch.bfloat16):
        for d, n_q, n_kv, new in ((128, 32, 8, 90), (128, 28, 4, 300), (256, 8, 4, 200)):
            gen = torch.Generator(device="cuda").manual_seed(d)
            g = KVArena(1, n_q, n_kv, d, 2048, 16, 400, dtype=dtype, sliding_popn_refuses=False)
            g.set_chunk_kernel(6)
            rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=dtype)
            seqs, ctx = [g.new_seq() for _ in range(3)], [37, 500, 1203]
            g.begin_step(seqs, ctx)
            k0, v0 = rand(sum(ctx) * n_kv * d), rand(sum(ctx) * n_kv * d)
            g.append(0, k0, v0)
            q, k, v = (rand(3 * new * h * d) for h in (n_q, n_kv, n_kv))
            g.begin_step(seqs, [new] * 3)
            out = g.attention(0, q, k, v, d ** -0.5)
            assert g.device_status() == 0
            # f64 reference
            off = ko = 0
            for c in ctx:
                K = torch.cat([k0.view(-1)[ko * n_kv * d:(ko + c) * n_kv * d].view(n_kv, c, d), k[off * n_kv * d:(off + new) * n_kv * d].view(n_kv, new, d)], 1).double()
                V = torch.cat([v0.view(-1)[ko * n_kv * d:(ko + c) * n_kv * d].view(n_kv, c, d), v[off * n_kv * d:(off + new) * n_kv * d].view(n_kv, new, d)], 1).double()
                Q = q[off * n_q * d:(off + new) * n_q * d].view(n_q, new, d).double()
                s = Q @ K.repeat_interleave(n_q // n_kv, 0).transpose(1, 2) * d ** -0.5
                s.masked_fill_(torch.arange(c + new, device="cuda")[None, :] > c + torch.arange(new, device="cuda")[:, None], -float("inf"))
                ref = s.softmax(-1) @ V.repeat_interleave(n_q // n_kv, 0)
                got = out[off * n_q * d:(off + new) * n_q * d].view(n_q, new, d).double()
                # outputs and probabilities are rounded to 8 (bf16) or 11 bits: 2^-9 and 2^-12 relative each, as rms
                # over many terms well below these
                assert (got - ref).norm() / ref.norm() < (2 ** -8 if dtype == torch.bfloat16 else 2 ** -10.5)
                off += new
                ko += c


def test_both_halves_of_a_row_see_the_same_maxima_over_many_tiles():
    # 512 tokens after 6000, nothing cut: 48 to 51 KV tiles per item, whose row maxima rise and move the reference nearly
    # every tile.  Every run has to give the same bits.
    from combsengine_b200 import KVArena
    n_q, n_kv, d, ctx, new = 32, 8, 128, 6000, 512
    gen = torch.Generator(device="cuda").manual_seed(7)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    g = KVArena(1, n_q, n_kv, d, 8192, 16, 512, sliding_popn_refuses=False)
    g.set_chunk_split(1)
    g.set_chunk_kernel(6)
    rise = lambda first, n: (0.1 * rand(n_kv * n * d).view(n_kv, n, d) + torch.arange(first, first + n, device="cuda")[None, :, None] / 128).half().view(-1)
    s = g.new_seq()
    g.begin_step([s], [ctx])
    g.append(0, rise(0, ctx), rand(ctx * n_kv * d))
    q, k, v = 0.1 * rand(new * n_q * d) + 1, rise(ctx, new), rand(new * n_kv * d)

    def run():
        g.begin_step([s], [new])
        out = g.attention(0, q, k, v, d ** -0.5)
        s.popn(new)
        return out

    first = run()
    for _ in range(60):
        assert torch.equal(run(), first)
    g.set_chunk_kernel(3)
    other = run()
    assert g.device_status() == 0
    assert (first.double() - other.double()).norm() <= 2 ** -9 * other.double().norm()  # P and the output rounded to 11 bits


@pytest.mark.parametrize("n_q,n_kv,d", [(28, 4, 128), (8, 4, 256)])
def test_int8_pages_on_pairs_of_sms(n_q, n_kv, d):
    # the kernel reads the float copy of the step's pages, through the copy's own maps
    p = Pair(1, n_q, n_kv, d, 2048, num_pages=400, seed=d, shuffle_free_list=True, quantize_kv=True, chunk_kernel=6)
    seqs = [p.new_seq() for _ in range(3)]
    p.step(seqs, [300, 17, 90])
    p.step(seqs, [129, 5, 700])
    p.step([seqs[1]], [40])
    p.assert_state_equal("used")


def test_pairs_are_refused_where_there_is_no_such_kernel():
    from combsengine_b200 import CbkvError, KVArena
    g = KVArena(1, 8, 2, 64, 256, 16, 16)
    with pytest.raises(CbkvError):
        g.set_chunk_kernel(6)
    for bad in (-1, 7):
        with pytest.raises(CbkvError):
            g.set_chunk_kernel(bad)


@pytest.mark.parametrize("n_q,n_kv,d,n_seqs,ctx,new,kernel", [
    (32, 8, 128, 1, 512, 512, 6), (28, 4, 128, 1, 400, 40, 6), (32, 8, 128, 4, 1024, 512, 3), (28, 4, 128, 8, 2000, 5, 3), (32, 8, 128, 64, 33, 2, 1),
    (8, 4, 256, 1, 512, 512, 6), (8, 4, 256, 1, 2000, 9, 6), (8, 4, 256, 16, 2000, 5, 2), (8, 4, 256, 64, 33, 5, 1)])
def test_the_default_takes_pairs_where_its_model_expects_them_to_end_sooner(n_q, n_kv, d, n_seqs, ctx, new, kernel):
    # on either side of the line the output is, bit for bit, that of the kernel which the rule names
    from combsengine_b200 import KVArena
    g = KVArena(1, n_q, n_kv, d, 4096, 16, n_seqs * 160, sliding_popn_refuses=False)
    gen = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    seqs = [g.new_seq() for _ in range(n_seqs)]
    g.begin_step(seqs, [ctx] * n_seqs)
    g.append(0, rand(n_seqs * ctx * n_kv * d), rand(n_seqs * ctx * n_kv * d))
    q, k, v = (rand(n_seqs * new * h * d) for h in (n_q, n_kv, n_kv))
    outs = {}
    for mode in (5, 1, 3 if d == 128 else 2, 6):
        g.set_chunk_kernel(mode)
        g.begin_step(seqs, [new] * n_seqs)
        assert mode != 5 or g.debug_chunk_choice()["kernel"] == kernel
        outs[mode] = g.attention(0, q, k, v, d ** -0.5)
        assert g.device_status() == 0
        for s in seqs:
            s.popn(new)
    same = [mode for mode in outs if mode != 5 and torch.equal(outs[mode], outs[5])]
    assert same == [kernel]
