"""Decode steps whose norm and rotation ride inside the decode kernel, against the same step in two calls (needs a B200)."""
import pytest
import torch

from combsengine_b200 import KVArena, QKNorm, RotaryEmbedding, attention_rope, rope_append

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norm", [None, "rms", "gemma"])
@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("n_q,n_kv,d,dtype", [(9, 3, 64, torch.float16), (28, 4, 128, torch.bfloat16), (8, 1, 128, torch.float16), (8, 4, 256, torch.bfloat16)])
def test_one_call_equals_rotate_and_append_then_attention(n_q, n_kv, d, dtype, int8, norm):
    # contexts that start a page, fill one, and are cut between CTAs; without a norm the same bits, with one the rows may
    # differ by a rounding (the sum of squares has no defined order): one ulp of the type in K, hence in the scores
    gen = torch.Generator(device="cuda").manual_seed(d)
    g = KVArena(1, n_q, n_kv, d, 4096, 16, 600, dtype=dtype, sliding_popn_refuses=False, quantize_kv=int8)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=dtype)
    rope = RotaryEmbedding(g, 500000.0, 4096)
    ctx = [1, 15, 16, 700, 3000]
    seqs = [g.new_seq() for _ in ctx]
    g.begin_step(seqs, ctx)
    g.append(0, rand(sum(ctx) * n_kv * d), rand(sum(ctx) * n_kv * d))
    qn = QKNorm(0.1 * rand(d), 0.1 * rand(d) + (0 if norm == "gemma" else 1), 1e-6, norm == "gemma") if norm else None
    q, k, v = (rand(len(ctx) * h * d) for h in (n_q, n_kv, n_kv))

    def pages():
        out = []
        for s in seqs:
            page = int(s.block_table()[-1])
            out += g.export_page_quant(0, page) if int8 else g.export_page(0, page)
        return out

    g.begin_step(seqs, [1] * len(ctx))
    one = attention_rope(g, 0, rope, q, k, v, d ** -0.5, norm=qn)
    one_pages = pages()
    for s in seqs:
        s.popn(1)
    g.begin_step(seqs, [1] * len(ctx))
    qr = rope_append(g, 0, rope, q, k, v, norm=qn)
    two = g.paged_attention(0, qr, d ** -0.5)
    assert g.device_status() == 0
    if norm is None:
        assert torch.equal(one, two)
        assert all((x == y).all() for x, y in zip(one_pages, pages()))
    else:
        ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
        assert (one.double() - two.double()).norm() <= 4 * ulp * two.double().norm()
    rope.close()
