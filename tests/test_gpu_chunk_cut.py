"""Chunk steps on the tcgen05 kernels against the oracle (needs a B200): steps of a few tokens and mixed steps at every
head_dim that the kernels take, items of one K/V tile and of many, cut along K/V and whole, with and without windows."""
import numpy as np
import pytest
import torch

from kvcase import Pair, assert_attention_close

pytestmark = pytest.mark.gpu

REPEATS = 40


def _inputs(p, pos, new, grow):
    """q, k, v of one layer, packed.  `grow`: K rows lengthen with their position and every query points along them, so a
    row's maximum rises by more than a factor 2^8 from one K/V tile to the next and O is rescaled; otherwise that is rare."""
    q, k, v = ([p.rand(h, n) for n in new] for h in (p.n_q, p.n_kv, p.n_kv))
    if grow:
        for i, (p0, n) in enumerate(zip(pos, new)):
            t = np.arange(p0, p0 + n, dtype=np.float32)[None, :, None] / 64
            k[i] = (0.1 * k[i].astype(np.float32) + t * 4 / np.sqrt(p.d)).astype(np.float16)
            q[i] = (0.1 * q[i].astype(np.float32) + 1).astype(np.float16)
    return [np.concatenate([x.reshape(-1) for x in xs]) for xs in (q, k, v)]


def _fill(p, pair, n, layers, grow):
    """n cached tokens, appended without attention."""
    p.g.begin_step([pair[0]], [n])
    p.o.batch_begin([pair[1]], [n])
    for l in layers:
        _, k, v = _inputs(p, [0], [n], grow)
        p.g.append(l, torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda())
        pair[1].append_only(l, k.reshape(p.n_kv, n, p.d), v.reshape(p.n_kv, n, p.d), 0)


def _step(p, pairs, new, layers, grow, repeats=REPEATS):
    """One step against the oracle, then rolled back and run again: every run has to give the same bits."""
    gs, os_ = [s[0] for s in pairs], [s[1] for s in pairs]
    pos, scale = [s.seq_len() for s in gs], p.d ** -0.5
    data = {l: _inputs(p, pos, new, grow) for l in layers}
    dev = {l: [torch.from_numpy(x).cuda() for x in data[l]] for l in layers}
    outs = []
    for r in range(repeats):
        p.g.begin_step(gs, new)
        outs.append([p.g.attention(l, *dev[l], scale) for l in layers])
        if r + 1 < repeats:
            for s, n in zip(gs, new):
                s.popn(n)
    assert p.g.device_status() == 0
    p.o.batch_begin(os_, new)
    for i, l in enumerate(layers):
        ref = p.o.batch_layer(os_, new, l, *data[l], p.n_q, scale, None)
        assert_attention_close(outs[0][i].cpu().numpy(), ref, f"layer {l} contexts {pos} new {new}")
        for r in range(1, repeats):
            assert torch.equal(outs[r][i], outs[0][i]), f"layer {l} contexts {pos} new {new}: run {r} differs"


KERNELS = [(9, 3, 64, 0), (28, 4, 128, 2), (28, 4, 128, 3), (28, 4, 128, 5), (28, 4, 128, 6), (8, 4, 256, 0), (8, 4, 256, 5), (8, 4, 256, 6)]  # q heads, kv heads, head_dim, chunk kernel


@pytest.mark.parametrize("grow", [False, True])
@pytest.mark.parametrize("n_q,n_kv,d,kernel", KERNELS)
def test_few_and_mixed_tokens_over_items_of_one_to_many_kv_tiles(n_q, n_kv, d, kernel, grow):
    # A layer with a window next to a global one.  K/V tiles hold 64 or 128 tokens: the contexts give items of 1, 2, 3, 4
    # and more tiles; alone, a long one is cut into short slices, in a batch into longer ones.
    p = Pair(2, n_q, n_kv, d, 8192, num_pages=1400, windows=[300, None], seed=d + kernel, shuffle_free_list=True,
             popn_refuses=False, chunk_kernel=kernel)
    for ctx in (1, 60, 126, 250, 380, 500, 2050):
        s = p.new_seq()
        _fill(p, s, ctx, [0, 1], grow)
        _step(p, [s], [5 if ctx % 4 else 2], [0, 1], grow)
    long = p.new_seq()
    _fill(p, long, 6100, [0, 1], grow)
    _step(p, [long], [9], [0, 1], grow)
    everyone = p.seqs
    _step(p, everyone, [5] * len(everyone), [0, 1], grow)
    _step(p, everyone, [1, 2, 3, 1, 140, 9, 1, 130], [0, 1], grow)  # two prompts' chunks among others' few tokens


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_cut_plans_of_two_windows_share_a_step(order):
    # 58 sequences of very different lengths: the layer with a window is cut into fewer slices of more items than the
    # global one, and each is launched again after the other.  Reference: the same step with nothing cut.
    from combsengine_b200 import KVArena
    ctx, new = [30000] * 15 + [1100] * 26 + [120] * 17, 5
    n_q, n_kv, d = 8, 4, 256
    g = KVArena(2, n_q, n_kv, d, 30016, 16, sum(c // 16 + 2 for c in ctx), [1024, None], sliding_popn_refuses=False)
    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    seqs = [g.new_seq() for _ in ctx]
    for s, c in zip(seqs, ctx):
        g.begin_step([s], [c])
        for l in range(2):
            g.append(l, rand(c * n_kv * d), rand(c * n_kv * d))
    q = [rand(len(ctx) * new * n_q * d) for _ in range(2)]
    kv = [[rand(len(ctx) * new * n_kv * d) for _ in range(2)] for _ in range(2)]
    outs = {}
    for parts in (64, 1):
        g.begin_step(seqs, [new] * len(ctx))
        if parts == 1:
            g.set_chunk_split(1)
        else:
            plans = [g.debug_tile_plan(w, 64, 64, 64) for w in (1024, 0)]
            assert plans[0]["n_cut"] > 148 > plans[1]["n_cut"] > 0 and plans[1]["n_slots"] > plans[0]["n_slots"] * 5 // 4
        for l in order:
            g.append(l, *kv[l])
        outs[parts] = [g.paged_attention(l, q[l], d ** -0.5) for l in order + order]
        assert g.device_status() == 0
        for s in seqs:
            s.popn(new)
    for cut, whole in zip(outs[64], outs[1]):
        assert_attention_close(cut.cpu().numpy(), whole.cpu().numpy(), f"order {order}")
    assert all(torch.equal(outs[64][i], outs[64][i + 2]) for i in range(2))


def _arena_with_context(d, ctx, seed=3, layers=1):
    from combsengine_b200 import KVArena
    g = KVArena(layers, 8, 2, d, 2048, 16, 400, sliding_popn_refuses=False)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    s = g.new_seq()
    g.begin_step([s], [ctx])
    for l in range(layers):
        g.append(l, rand(ctx * 2 * d), rand(ctx * 2 * d))
    return g, s, rand


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("new", [5, 200])
def test_queries_and_outputs_at_any_element_address(d, new):
    # the tensor-core kernels move 16 bytes at a time; q at a multiple of 4 bytes and out at any element take the other one
    g, s, rand = _arena_with_context(d, 700)
    q, k, v = (rand(new * h * d) for h in (8, 2, 2))
    outs = []
    for q_off, out_off in ((0, 0), (2, 0), (0, 1), (6, 3)):
        qv = torch.empty(q.numel() + 8, dtype=q.dtype, device="cuda")[q_off:q_off + q.numel()].copy_(q)
        out = torch.zeros(q.numel() + 8, dtype=q.dtype, device="cuda")[out_off:out_off + q.numel()]
        g.begin_step([s], [new])
        outs.append(g.attention(0, qv, k, v, d ** -0.5, out=out).cpu().numpy())
        assert g.device_status() == 0
        s.popn(new)
    for o in outs[1:]:
        assert_attention_close(o, outs[0])


@pytest.mark.parametrize("d", [64, 128, 256])
def test_scale_that_vanishes_in_32_bits(d):
    # every visible key gets the same weight; masked scores stay masked
    p = Pair(1, 8, 2, d, 512, seed=d)
    s = p.new_seq()
    p.step([s], [70], scale=1e-50)
    p.step([s], [5], scale=1e-50)
    p.step([s], [5], scale=1e-44)


def test_the_cut_can_be_set_back_to_its_default():
    from combsengine_b200 import CbkvError
    g, s, rand = _arena_with_context(128, 1500)
    q, k, v = (rand(5 * h * 128) for h in (8, 2, 2))
    outs = []
    for parts in (None, 1, 8, 64):
        if parts:
            g.set_chunk_split(parts)
        g.begin_step([s], [5])
        outs.append(g.attention(0, q, k, v, 0.1))
        s.popn(5)
    assert torch.equal(outs[0], outs[3])  # the same slices, summed in the same order
    for o in outs[1:3]:
        assert_attention_close(o.cpu().numpy(), outs[0].cpu().numpy())
    for bad in (0, 65):
        with pytest.raises(CbkvError):
            g.set_chunk_split(bad)


@pytest.mark.parametrize("overlap", [True, False])
@pytest.mark.parametrize("d,int8", [(64, False), (128, False), (128, True)])
def test_overlap_switch_covers_every_launch_of_a_chunk_step(d, int8, overlap):
    # captured into a graph that is not run: launches that may overlap are joined by programmatic edges
    import ctypes as C
    from combsengine_b200 import KVArena, RotaryEmbedding, attention_rope
    rt = C.CDLL("libcudart.so.12")
    g = KVArena(1, 8, 2, d, 256, 16, 40, quantize_kv=int8)
    g.set_decode_tuning(overlap_launches=overlap)
    g.set_chunk_kernel(3 if d == 128 else 2)  # the mma.sync kernel is never launched early
    rope = RotaryEmbedding(g, 10000.0, 256)
    s = g.new_seq()
    q, k, v = (torch.randn(70 * h * d, device="cuda").half() for h in (8, 2, 2))
    out = torch.empty_like(q)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    g.begin_step([s], [70], stream=stream)

    def calls():
        g.attention(0, q, k, v, 0.1, out=out, stream=stream)
        attention_rope(g, 0, rope, q, k, v, 0.1, out=out, stream=stream)

    calls()  # uploads, plans and workspaces are in place after this
    st, graph, n = C.c_void_p(stream.cuda_stream), C.c_void_p(), C.c_size_t()
    assert rt.cudaStreamBeginCapture(st, 2) == 0  # relaxed
    calls()
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0
    assert rt.cudaGraphGetEdges_v2(graph, None, None, None, C.byref(n)) == 0
    ends, data = [(C.c_void_p * n.value)() for _ in range(2)], (C.c_ubyte * 8 * n.value)()  # from port, to port, type, padding
    assert rt.cudaGraphGetEdges_v2(graph, *ends, data, C.byref(n)) == 0
    assert n.value == (6 if int8 else 3)
    assert [e[2] for e in data] == [1 if overlap else 0] * n.value
    assert rt.cudaGraphDestroy(graph) == 0
    torch.cuda.synchronize()
    assert g.device_status() == 0
    rope.close()


@pytest.mark.parametrize("n_q,n_kv,d,tcgen05,n_seqs,ctx,new,mma", [
    (32, 8, 128, 3, 64, 33, 2, True), (32, 8, 128, 3, 18, 33, 2, False), (32, 8, 128, 3, 64, 600, 2, True), (32, 8, 128, 3, 32, 600, 2, False),
    (28, 4, 128, 3, 1, 1, 40, True), (28, 4, 128, 3, 1, 400, 40, False), (8, 4, 256, 2, 64, 33, 5, True), (8, 4, 256, 2, 64, 900, 5, False),
    (9, 3, 64, 2, 64, 33, 5, False)])
def test_many_short_sequences_take_the_mma_kernel(n_q, n_kv, d, tcgen05, n_seqs, ctx, new, mma):
    # on either side of the line the output is, bit for bit, that of the kernel which the rule names
    from combsengine_b200 import KVArena
    g = KVArena(1, n_q, n_kv, d, 1024, 16, n_seqs * 64, sliding_popn_refuses=False)
    gen = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    seqs = [g.new_seq() for _ in range(n_seqs)]
    g.begin_step(seqs, [ctx] * n_seqs)
    g.append(0, rand(n_seqs * ctx * n_kv * d), rand(n_seqs * ctx * n_kv * d))
    q, k, v = (rand(n_seqs * new * h * d) for h in (n_q, n_kv, n_kv))
    outs = {}
    for kernel in (0, 1, tcgen05):
        g.set_chunk_kernel(kernel)
        g.begin_step(seqs, [new] * n_seqs)
        outs[kernel] = g.attention(0, q, k, v, d ** -0.5)
        assert g.device_status() == 0
        for s in seqs:
            s.popn(new)
    assert not torch.equal(outs[1], outs[tcgen05])
    assert torch.equal(outs[0], outs[1 if mma else tcgen05])
    assert_attention_close(outs[0].cpu().numpy(), outs[tcgen05 if mma else 1].cpu().numpy())


@pytest.mark.parametrize("n_q,n_kv,d,int8,pages,uncut", [
    (9, 3, 64, False, 40, True), (9, 3, 64, False, 41, False), (32, 8, 128, False, 40, True), (32, 8, 128, False, 41, False),
    (8, 4, 256, False, 16, True), (8, 4, 256, False, 24, False), (32, 8, 128, True, 16, True), (32, 8, 128, True, 24, False)])
def test_short_decode_is_cut_where_that_is_faster(n_q, n_kv, d, int8, pages, uncut):
    # one CTA per (sequence, kv head), asked for by the CTA limit, gives the same bits as the default where nothing is cut
    from combsengine_b200 import KVArena
    g = KVArena(1, n_q, n_kv, d, 1024, 16, 128, quantize_kv=int8)
    gen = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
    seqs = [g.new_seq() for _ in range(2)]
    n = 16 * pages - 3
    g.begin_step(seqs, [n] * 2)
    g.append(0, rand(2 * n * n_kv * d), rand(2 * n * n_kv * d))
    q, k, v = (rand(2 * h * d) for h in (n_q, n_kv, n_kv))
    outs = []
    for max_ctas in (0, 2 * n_kv):
        g.set_decode_tuning(max_ctas=max_ctas)
        g.begin_step(seqs, [1] * 2)
        outs.append(g.attention(0, q, k, v, d ** -0.5))
        for s in seqs:
            s.popn(1)
    assert g.device_status() == 0
    assert torch.equal(outs[0], outs[1]) == uncut
    assert_attention_close(outs[0].cpu().numpy(), outs[1].cpu().numpy())
