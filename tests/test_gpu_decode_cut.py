"""Decode launches whose CTAs hold one segment each (ranges that end where segments do, short segments uncut, the last piece
combined by all warps) against attention in float64, at the sizes where the plan changes."""
import pytest
import torch

from combsengine_b200 import KVArena

pytestmark = pytest.mark.gpu


def reference(q, k, v, scale, window):
    """q (n_q, d), k and v (n_kv, tokens, d), float64: one token's attention."""
    n_kv, t, d = k.shape
    if window:
        k, v = k[:, max(0, t - window):], v[:, max(0, t - window):]
    s = q.view(n_kv, -1, d) @ k.transpose(1, 2) * scale
    return (s.softmax(-1) @ v).reshape(-1, d)


def quantised(x):
    g = x.to(torch.float32).reshape(-1, 32)
    s = (g.abs().amax(1, keepdim=True) / 127).clamp(min=1e-8)
    return ((g / s).round().clamp(-127, 127) * s.to(x.dtype).to(torch.float32)).view(x.shape)


# lengths after the step: one page and a page more, the longest segment that is not cut and one page more, several rounds of
# the ring, unequal ones (ranges of 6 pages up to the whole segment), and a segment count that fills the chip
@pytest.mark.parametrize("d,n_kv,n_rep,int8", [(64, 3, 3, False), (128, 8, 4, False), (128, 4, 7, False), (256, 4, 2, False), (64, 3, 3, True), (128, 4, 7, True), (256, 4, 2, True)])
@pytest.mark.parametrize("lens,window", [([1, 16, 17], None), ([272, 273], None), ([384, 385], None), ([448], None), ([449], None), ([320, 321], None),
                                         ([1500, 40, 700], None), ([3000, 1000], 1024), ([100 + 37 * i for i in range(20)], None), ([900] * 36, None)])
def test_one_segment_per_cta(d, n_kv, n_rep, int8, lens, window):
    check(d, n_kv, n_rep, int8, lens, window, 4)


# arenas of one layer keep longer segments whole, those of two do not
@pytest.mark.parametrize("layers", [1, 2])
@pytest.mark.parametrize("d,n_kv,n_rep", [(64, 3, 3), (128, 4, 7), (128, 1, 4)])
@pytest.mark.parametrize("lens", [[384, 385], [448, 449], [640], [641, 300], [640] * 20])
def test_arenas_of_few_layers(d, n_kv, n_rep, lens, layers):
    check(d, n_kv, n_rep, False, lens, None, layers)


def check(d, n_kv, n_rep, int8, lens, window, layers):
    dt, n_q, B = torch.float16, n_kv * n_rep, len(lens)
    torch.manual_seed(sum(lens) + d)
    a = KVArena(layers, n_q, n_kv, d, max(lens) + 16, 16, sum(-(-n // 16) for n in lens) + 4, [window] * layers, dt, sliding_popn_refuses=False, quantize_kv=int8)
    a.set_free_list(torch.randperm(a.num_pages).numpy())
    seqs = [a.new_seq() for _ in lens]
    kv = [torch.randn(2, n_kv, n, d, device="cuda", dtype=dt) for n in lens]
    old = [(s, x) for s, x in zip(seqs, kv) if x.shape[2] > 1]
    if old:
        a.begin_step([s for s, _ in old], [x.shape[2] - 1 for _, x in old])
        a.append(0, *[torch.cat([x[i, :, :-1].reshape(-1) for _, x in old]) for i in range(2)])
    q = torch.randn(B, n_q, d, device="cuda", dtype=dt)
    k, v = (torch.cat([x[i, :, -1].reshape(-1) for x in kv]) for i in range(2))
    a.begin_step(seqs, [1] * B)
    out = torch.zeros_like(q)
    a.attention(0, q.view(-1), k, v, d ** -0.5, out=out.view(-1))
    again = torch.zeros_like(q)
    a.paged_attention(0, q.view(-1), d ** -0.5, out=again.view(-1))  # the new row is in its page by now
    assert a.device_status() == 0
    for b in range(B):
        x = (quantised(kv[b]) if int8 and window is None else kv[b]).to(torch.float64)
        ref = reference(q[b].to(torch.float64), x[0], x[1], d ** -0.5, window)
        for o in (out[b], again[b]):
            err = (o.to(torch.float64) - ref).abs()
            assert bool((err <= 2e-3 + 1e-2 * ref.abs()).all()), (b, lens[b], float(err.max()))
    a.close()


# A layer with a window of its own keeps 16-bit pages in an arena of int8 ones, and an int8 layer may be called with the same
# window: each has its own cut, whichever comes first in the step (16-bit segments of 16 or 24 pages stay whole, int8 ones are cut).
@pytest.mark.parametrize("d,consumers,n", [(256, 0, 251), (128, 6, 380)])
def test_layers_of_both_kinds_under_one_window(d, consumers, n):
    n_kv, n_q, dt, window, ctx = 4, 8, torch.float16, 512, [n, n - 11]
    torch.manual_seed(d)
    a = KVArena(4, n_q, n_kv, d, 1024, 16, 64, [window, None, None, None], dt, sliding_popn_refuses=False, quantize_kv=True)
    a.set_decode_tuning(consumers=consumers)
    seqs = [a.new_seq() for _ in ctx]
    rand = lambda n: torch.randn(n, device="cuda", dtype=dt)
    a.begin_step(seqs, ctx)
    for layer in range(2):
        a.append(layer, rand(sum(ctx) * n_kv * d), rand(sum(ctx) * n_kv * d))
    q, k, v = (rand(2 * h * d) for h in (n_q, n_kv, n_kv))
    outs = []
    for order in ((0,), (1,), (0, 1), (1, 0)):
        a.begin_step(seqs, [1, 1])
        outs.append({layer: a.attention(layer, q, k, v, d ** -0.5, window=window) for layer in order})
        for s in seqs:
            s.popn(1)
    assert a.device_status() == 0
    for both in outs[2:]:
        for layer in range(2):
            assert torch.equal(both[layer], outs[layer][layer])
    a.close()


@pytest.mark.parametrize("d,int8", [(64, False), (128, False), (256, False), (128, True)])
def test_no_more_ctas_are_planned_than_run_at_a_time(d, int8):
    # two CTAs per SM asked for: the cut is that of one where the kernel has the registers of one
    n_kv, n_q, dt, ctx = 4, 8, torch.float16, [900 + 61 * i for i in range(40)]
    torch.manual_seed(d)
    a = KVArena(3, n_q, n_kv, d, max(ctx) + 16, 16, sum(n // 16 + 2 for n in ctx), None, dt, quantize_kv=int8)
    seqs = [a.new_seq() for _ in ctx]
    rand = lambda n: torch.randn(n, device="cuda", dtype=dt)
    a.begin_step(seqs, ctx)
    a.append(0, rand(sum(ctx) * n_kv * d), rand(sum(ctx) * n_kv * d))
    q, k, v = (rand(len(ctx) * h * d) for h in (n_q, n_kv, n_kv))
    sms, outs = torch.cuda.get_device_properties(0).multi_processor_count, []
    for per_sm, max_ctas in ((1, 0), (2, 0), (2, sms)):
        a.set_decode_tuning(ctas_per_sm=per_sm, max_ctas=max_ctas)
        a.begin_step(seqs, [1] * len(ctx))
        outs.append(a.attention(0, q, k, v, d ** -0.5))
        for s in seqs:
            s.popn(1)
    assert a.device_status() == 0
    assert torch.equal(outs[0], outs[2])
    assert torch.equal(outs[0], outs[1]) != int8  # int8 pages: two run at a time, and the launch is cut for them
    a.close()


def test_the_plan_that_is_shown_follows_the_arenas_split():
    a = KVArena(3, 8, 4, 128, 8192, 16, 2048)
    seqs = [a.new_seq() for _ in range(4)]
    a.begin_step(seqs, [6000, 300, 4000, 2000])
    a.begin_step(seqs, [1] * 4)
    assert a.debug_decode_choice()["n_items"] == a.debug_decode_choice()["n_ctas"]
    a.set_decode_split(tail_pct=25, min_item=2)
    shown, asked = a.debug_decode_choice(), a.debug_decode_plan(0, 148, 25, 2)
    assert shown["n_items"] > shown["n_ctas"]
    assert (shown["items"] == asked["items"]).all() and (shown["segs"] == asked["segs"]).all()
    a.close()
