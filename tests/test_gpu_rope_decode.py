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


@pytest.mark.parametrize("n_kv,d,int8,norm,per_sm", [
    (8, 64, False, True, 3), (8, 64, True, True, 3), (8, 128, False, True, 2), (8, 128, True, True, 1), (8, 128, True, False, 5),
    (4, 256, False, True, 1), (4, 256, True, False, 1), (4, 256, True, True, 0), (8, 128, False, False, None)])
def test_rotation_rides_along_up_to_the_segments_per_sm_that_it_is_faster_for(n_kv, d, int8, norm, per_sm):
    # one launch per layer below the line, rotate-and-append or rotation and attention above it.  The outputs of a sequence
    # differ by the order of 32-bit sums, because one sequence more moves the cuts between CTAs: the neighbouring f16 value
    # at most, 2^-10 of it; with a norm by a rounding of the normed rows as well, as above
    from combsengine_b200 import kv
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = 2 * sms // n_kv if per_sm is None else per_sm * sms // n_kv
    gen = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    g = KVArena(2, 2 * n_kv, n_kv, d, 64, 16, 4 * (line + 1), sliding_popn_refuses=False, quantize_kv=int8)
    rope = RotaryEmbedding(g, 500000.0, 64)
    qn = QKNorm(0.1 * rand(d) + 1, 0.1 * rand(d) + 1, 1e-6, False) if norm else None
    seqs = [g.new_seq() for _ in range(line + 1)]
    g.begin_step(seqs, [20] * len(seqs))
    for l in range(2):
        g.append(l, rand(20 * len(seqs) * n_kv * d), rand(20 * len(seqs) * n_kv * d))
    q, k, v = (rand(len(seqs) * h * d) for h in (2 * n_kv, n_kv, n_kv))
    outs = []
    for n in ([line] if line else []) + [line + 1]:
        g.begin_step(seqs[:n], [1] * n)
        a = [x[:n * x.numel() // len(seqs)].contiguous() for x in (q, k, v)]
        attention_rope(g, 0, rope, *a, d ** -0.5, norm=qn)
        before = kv.launch_count()
        outs.append(attention_rope(g, 1, rope, *a, d ** -0.5, norm=qn))
        assert kv.launch_count() - before == (1 if n <= line or per_sm is None else 2)
        for s in seqs[:n]:
            s.popn(1)
    assert g.device_status() == 0
    for o in outs[1:]:
        x, y = outs[0].double(), o[:outs[0].numel()].double()
        assert (x - y).norm() <= 2.0 ** (-9 if norm else -10) * y.norm()
    rope.close()
