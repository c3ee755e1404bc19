"""Decode launches whose CTAs hold one segment each (ranges that end where segments do, short segments uncut, rings of the
ranges' size, the last piece combined by all warps) against attention in float64, at the sizes where the plan changes."""
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
    dt, n_q, B = torch.float16, n_kv * n_rep, len(lens)
    torch.manual_seed(sum(lens) + d)
    a = KVArena(4, n_q, n_kv, d, max(lens) + 16, 16, sum(-(-n // 16) for n in lens) + 4, [window] * 4, dt, sliding_popn_refuses=False, quantize_kv=int8)
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
