"""Host logic through the C ABI, no GPU: the manager against the reference's
known-answer tests (kv.rs:1075-1192) and against the oracle on random histories,
the decode work split, and the boundary itself (symbols, loud failure)."""
import ctypes as C
import os
import re

import numpy as np
import pytest
import torch

from combsengine_b200 import CbkvError, KVArena, _lib
from oracle import OracleArena

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def arena(max_seq_len=64, page_size=16, layers=2, num_pages=0, windows=None, **kw):
    return KVArena(layers, 4, 2, 64, max_seq_len, page_size, num_pages, windows, **kw)


def grow(a, s, total):  # the reference tests' grow() helper, kv.rs:1134-1137
    a.begin_step_host_only([s], [total - s.seq_len()])


def test_library_exports_every_declared_symbol():
    header = open(os.path.join(ROOT, "include", "combs_kv.h")).read()
    declared = set(re.findall(r"\b(cbkv_[a-z0-9_]+)\s*\(", header))
    assert declared, "no declarations found"
    lib = C.CDLL(_lib.LIB_PATH)
    for name in sorted(declared):
        assert hasattr(lib, name), f"{name} declared in include/combs_kv.h but not exported"
    assert declared == set(_lib.PROTOTYPES), "ctypes prototypes and header disagree"


def test_allocator_order_lifo_reset():  # kv.rs:1075-1107
    a = arena(48)
    s = a.new_seq()
    assert a.num_free_pages() == 3
    grow(a, s, 48)
    assert list(s.block_table()) == [0, 1, 2] and a.num_free_pages() == 0
    with pytest.raises(CbkvError, match="capacity exceeded"):
        grow(a, s, 49)
    assert s.popn(48) == 48
    assert list(a.free_list()) == [2, 1, 0]  # pushed in table.pop() order
    grow(a, s, 32)
    assert list(s.block_table()) == [0, 1]
    s.reset()
    assert a.num_free_pages() == 3 and list(a.free_list()) == [2, 1, 0]


def test_exhaustion_is_all_or_nothing():  # kv.rs:552-555
    a = arena(64, num_pages=3)
    s, t = a.new_seq(), a.new_seq()
    grow(a, s, 32)
    with pytest.raises(CbkvError, match="page allocator exhausted") as e:
        a.begin_step_host_only([s, t], [1, 17])
    assert e.value.code == -3
    assert s.seq_len() == 32 and t.seq_len() == 0 and a.num_free_pages() == 1


@pytest.mark.parametrize("n,pages", [(16, 1), (17, 2), (1, 1)])
def test_num_pages_rounds_up(n, pages):  # kv.rs:1109-1114
    assert arena(n).num_free_pages() == pages


def test_popn_frees_only_fully_unused_pages():  # kv.rs:1139-1160
    a = arena()
    c = a.new_seq()
    grow(a, c, 40)
    assert c.pages_used() == 3 and a.num_free_pages() == 1
    c.popn(9)
    assert (c.seq_len(), c.pages_used(), a.num_free_pages()) == (31, 2, 2)
    c.popn(15)
    assert c.pages_used() == 1
    c.popn(1)
    assert c.pages_used() == 1
    assert c.popn(1000) == 15
    assert (c.seq_len(), c.pages_used(), a.num_free_pages()) == (0, 0, 4)


def test_popn_boundary_and_regrowth_and_reset():  # kv.rs:1162-1192
    a = arena()
    c = a.new_seq()
    grow(a, c, 32)
    c.popn(16)
    assert c.pages_used() == 1 and a.num_free_pages() == 3
    c.popn(16)
    assert c.pages_used() == 0 and a.num_free_pages() == 4
    grow(a, c, 40)
    freed = c.block_table()[2]
    c.popn(9)
    grow(a, c, 33)
    assert c.pages_used() == 3 and a.num_free_pages() == 1 and c.block_table()[2] == freed
    c.reset()
    assert (c.seq_len(), c.pages_used(), a.num_free_pages()) == (0, 0, 4)


def test_errors_carry_the_reference_messages():
    a = arena(8, 4)
    s = a.new_seq()
    with pytest.raises(CbkvError, match=r"paged cache capacity exceeded: 9 > 8") as e:  # tests/kv_cache.rs:167-173
        a.begin_step_host_only([s], [9])
    assert e.value.code == -2 and s.seq_len() == 0
    with pytest.raises(CbkvError, match="dense contiguous appends") as e:  # kv.rs:671-674
        a.begin_step_host_only([s], [2], [3])
    assert e.value.code == -1
    with pytest.raises(CbkvError, match="sliding window must be >= 2, got 1"):  # kv.rs:514-516
        arena(windows=[1, None])
    with pytest.raises(CbkvError, match="one window entry per layer"):  # kv.rs:513
        arena(windows=[4])


def test_sliding_popn_refusal_rule():  # kv.rs:812-816, 1061-1073
    a = arena(64, windows=[4, None])
    s = a.new_seq()
    grow(a, s, 3)
    assert s.popn(1) == 1  # nothing evicted yet (seq_len <= w - 1)
    grow(a, s, 6)
    assert s.popn(1) == 0 and s.seq_len() == 6
    assert s.popn(0) == 0
    b = arena(64, windows=[4, None], sliding_popn_refuses=False)
    t = b.new_seq()
    grow(b, t, 6)
    assert t.popn(1) == 1


def test_page_stats_fields():  # kv.rs:535-546
    a = arena(64, windows=[None, 8])
    s = a.new_seq()
    grow(a, s, 20)
    st = s.page_stats()
    assert (st.pages_used, st.pages_free, st.num_pages, st.page_size, st.seq_len) == (2, 2, 4, 16, 20)
    assert (st.layers_materialized, st.layers_total, st.layers_sliding) == (0, 2, 0)
    assert a.page_bytes() == 16 * 2 * 64 * 2 * 2 * 2  # engine.rs:475-498


def test_prefix_sharing_refcounts_and_guards():
    a = arena(256, num_pages=16)
    p = a.new_seq()
    grow(a, p, 40)
    with pytest.raises(CbkvError, match="whole pages"):
        p.fork_prefix(20)
    c = p.fork_prefix(32)
    assert c.seq_len() == 32 and list(c.block_table()) == list(p.block_table()[:2])
    assert [a.refcount(int(x)) for x in p.block_table()] == [2, 2, 1]
    grow(a, c, 33)  # the child's first append takes a fresh page
    assert c.block_table()[2] not in p.block_table()
    assert c.popn(10) == 0  # would end inside a shared page
    assert c.popn(1) == 1 and c.pages_used() == 2
    free_before = a.num_free_pages()
    c.close()  # shared pages stay with the parent
    assert a.num_free_pages() == free_before
    assert [a.refcount(int(x)) for x in p.block_table()] == [1, 1, 1]


def random_history(seed, rolling=False):
    """The same random allocate/append/popn/fork/destroy/reset history on the manager and the oracle."""
    rng = np.random.default_rng(seed)
    pages = 96
    a = KVArena(2, 4, 2, 64, 400, 16, pages, sliding_popn_refuses=False)
    o = OracleArena(2, 2, 64, 400, 16, pages, rolling=False, dtype="f16")
    perm = rng.permutation(pages)
    a.set_free_list(perm)
    o.set_free_list(perm)
    seqs = []
    for step in range(300):
        op = rng.integers(0, 10)
        if op <= 1 and len(seqs) < 10:
            seqs.append((a.new_seq(), o.new_seq()))
        elif op <= 5 and seqs:
            idx = rng.permutation(len(seqs))[: rng.integers(1, len(seqs) + 1)]
            new = [int(rng.integers(1, 40)) for _ in idx]
            ok = True
            try:
                a.begin_step_host_only([seqs[i][0] for i in idx], new)
            except CbkvError as e:
                ok = False
                code = e.code
            if ok:
                o.batch_begin([seqs[i][1] for i in idx], new)
            else:
                with pytest.raises(Exception):
                    o.batch_begin([seqs[i][1] for i in idx], new)
                # the oracle is not all-or-nothing across a batch; rebuild it from the manager's state
                return None if code == 0 else "diverged-on-error"
        elif op == 6 and seqs:
            i = rng.integers(len(seqs))
            n = int(rng.integers(0, 50))
            assert seqs[i][0].popn(n) == seqs[i][1].popn(n)
        elif op == 7 and seqs:
            i = rng.integers(len(seqs))
            n = (seqs[i][0].seq_len() // 16) * 16
            if n and len(seqs) < 10:
                n = int(rng.integers(1, n // 16 + 1)) * 16
                seqs.append((seqs[i][0].fork_prefix(n), seqs[i][1].fork_prefix(n)))
        elif op == 8 and seqs:
            i = rng.integers(len(seqs))
            s, t = seqs.pop(i)
            s.close(); t.close()
        elif op == 9 and seqs and rng.integers(4) == 0:
            i = rng.integers(len(seqs))
            seqs[i][0].reset(); seqs[i][1].reset()
        assert list(a.free_list()) == list(o.free_list()), step
        for s, t in seqs:
            assert s.seq_len() == t.seq_len()
            assert list(s.block_table()) == list(t.block_table())
        for pg in range(pages):
            assert a.refcount(pg) == o.refcount(pg)
    return "done"


@pytest.mark.parametrize("seed", range(6))
def test_manager_matches_oracle_on_random_histories(seed):
    random_history(seed)


@pytest.mark.parametrize("window,n_ctas,tail_pct,min_item", [(0, 1, -1, -1), (0, 7, -1, -1), (0, 148, -1, -1), (0, 148, 40, 4),
                                                              (0, 296, 25, 0), (0, 5000, -1, -1), (100, 13, -1, -1),
                                                              (1024, 148, -1, 2), (17, 64, -1, -1)])
def test_decode_plan_covers_every_page_once(window, n_ctas, tail_pct, min_item):
    rng = np.random.default_rng(window + n_ctas)
    a = KVArena(1, 28, 4, 128, 5000, 16, 20000)
    seqs = [a.new_seq() for _ in range(24)]
    lens = [int(x) for x in rng.integers(1, 4100, len(seqs))]
    lens[0], lens[1], lens[2] = 2, 16, 17  # lengths after the decode step
    a.begin_step_host_only(seqs, [n - 1 for n in lens])   # the cached prefix
    a.begin_step_host_only(seqs, [1] * len(seqs))         # the decode step being split
    L = [s.seq_len() for s in seqs]
    pl = a.debug_decode_plan(window, n_ctas, tail_pct, min_item)
    Hkv = 4
    segs, items = pl["segs"], pl["items"]
    assert pl["n_segs"] == len(seqs) * Hkv and pl["n_items"] == pl["n_ctas"] * pl["levels"]
    sub = segs[:, 0]
    assert sub[0] == 0 and sub[-1] == pl["n_units"]
    # segments: the visible pages of every (sequence, kv head)
    tok = 0
    for b, n in enumerate(L):
        q = n - 1
        lo = max(0, q - window + 1) if window else 0
        for h in range(Hkv):
            s = b * Hkv + h
            assert segs[s, 1] == lo // 16 and segs[s, 2] == q and segs[s, 3] == tok
            assert sub[s + 1] - sub[s] == q // 16 - lo // 16 + 1
        tok += 1
    # items: non-empty, disjoint, and together exactly the units
    assert np.all(items[:, 1] > items[:, 0])
    order = np.argsort(items[:, 0], kind="stable")
    srt = items[order]
    assert srt[0, 0] == 0 and srt[-1, 1] == pl["n_units"] and np.array_equal(srt[1:, 0], srt[:-1, 1])
    # claim order: a CTA's first item is the head of its range, and later levels never grow
    G, J = pl["n_ctas"], pl["levels"]
    size = (items[:, 1] - items[:, 0]).reshape(J, G)
    if J > 1:
        assert size[0].min() >= size[1:].max()
        assert np.all(size[1:-1].min(axis=1) + 1 >= size[2:].max(axis=1)) if J > 2 else True
    # a CTA's first item is a function of the launch totals alone (the kernel computes it instead of reading it)
    U, pct = pl["n_units"], (25 if tail_pct < 0 else tail_pct) if J > 1 else 0
    for c in range(G):
        rb, re = U * c // G, U * (c + 1) // G
        assert items[c, 0] == rb and items[c, 1] == re - (re - rb) * pct // 100
    per_range = size.sum(axis=0)
    assert per_range.max() - per_range.min() <= 1  # balanced to one page before any claiming
    # parts: every segment knows how many items touch it, and every item its place among them
    parts = 0
    for s in range(pl["n_segs"]):
        touching = [i for i in order if items[i, 0] < sub[s + 1] and items[i, 1] > sub[s]]
        assert segs[s, 4] == len(touching)
        if len(touching) > 1:
            assert segs[s, 5] == parts
            parts += len(touching)
        else:
            assert segs[s, 5] == -1
        for rank, i in enumerate(touching):
            if sub[s] <= items[i, 0] < sub[s + 1]:
                assert items[i, 2] == s and items[i, 3] == rank
            else:
                assert rank == 0  # an item that runs into a segment from before it is that segment's part 0
    assert parts == pl["n_parts"]


@pytest.mark.parametrize("d,int8,lens,window", [
    (64, False, [385, 300, 20], 0), (64, False, [384, 300, 20], 0), (128, False, [449], 0), (128, False, [448, 448], 0),   # uncut or not
    (128, False, [300, 800, 1400, 2000], 0), (256, False, [1001, 3000], 0), (256, False, [8192] * 16, 1024),
    (128, True, [300, 2000, 17, 5000], 0), (256, True, [193, 192], 0), (128, False, [5] * 37, 0), (128, False, [5] * 38, 0),
    (128, False, [32000] + [40] * 30, 0), (64, False, [1, 16, 17], 0),
    # nearly as many segments as CTAs, one sequence longer than the others: at the line and past it
    (64, False, [80] * 36 + [1136], 0), (64, False, [80] * 36 + [1216], 0), (128, True, [80] * 73 + [352], 0), (128, True, [80] * 73 + [480], 0)])
def test_decode_ranges_end_where_segments_do_when_that_costs_little(d, int8, lens, window):
    Hkv, C = 4, 4 if int8 and d <= 128 else 6
    most = 296 if int8 and d <= 128 else 148
    slack = {64: 20, 128: 16, 256: 8}[d] if int8 else {64: 64, 128: 48, 256: 16}[d]
    uncut = {64: 19, 128: 20, 256: 12}[d] if int8 else {64: 24, 128: 28, 256: 17}[d]
    a = KVArena(4, 8, Hkv, d, 33000, 16, 1 << 15)
    seqs = [a.new_seq() for _ in lens]
    if max(lens) > 1:
        old = [(s, n - 1) for s, n in zip(seqs, lens) if n > 1]
        a.begin_step_host_only([s for s, _ in old], [n for _, n in old])
    a.begin_step_host_only(seqs, [1] * len(seqs))
    pl = a.debug_decode_choice(window, int8, C, most)
    sub, items, U = pl["segs"][:, 0], pl["items"], pl["n_units"]
    pages = np.diff(sub)
    size = items[:, 1] - items[:, 0]
    assert pl["n_ctas"] == pl["n_items"] == len(items) <= most and size.min() >= 1
    assert items[0, 0] == 0 and items[-1, 1] == U and np.array_equal(items[1:, 0], items[:-1, 1])
    first = np.searchsorted(sub, items[:, 0], side="right") - 1
    aligned = bool(np.all(items[:, 1] <= sub[first + 1]))
    even = -(-U // min(most, max(1, -(-U // C))))
    limit = max(even, pages.max() if pages.max() <= uncut else C) + slack
    # ranges of at most `limit` pages that end where segments do exist exactly when the library takes such
    possible = int(np.sum(-(-pages // min(limit, pages.max())))) <= most
    assert aligned == possible or (aligned and pl["n_ctas"] == -(-U // even))
    if possible:
        assert size.max() <= limit
        if pages.max() <= uncut:
            assert len(items) == len(pages)
        for s in range(len(pages)):
            mine = np.flatnonzero(first == s)
            assert pl["segs"][s, 4] == len(mine) and np.ptp(size[mine]) <= 1
            assert np.array_equal(items[mine, 2], np.full(len(mine), s)) and np.array_equal(items[mine, 3], np.arange(len(mine)))
    assert pl["n_parts"] == int(np.sum(pl["segs"][:-1, 4][pl["segs"][:-1, 4] > 1]))


# the longest segments that stay whole: one layer (up to 16 segments of 16-bit pages, head_dim up to 128), two, and more
@pytest.mark.parametrize("layers", [1, 2, 3])
@pytest.mark.parametrize("d,int8,n_kv,seqs,one,more", [(64, False, 3, 2, 40, 24), (128, False, 8, 2, 40, 28), (128, False, 8, 3, 28, 28), (128, False, 1, 4, 40, 28),
                                                       (256, False, 4, 1, 17, 17), (64, True, 3, 2, 19, 19), (128, True, 4, 1, 20, 20), (256, True, 4, 1, 12, 12)])
def test_short_segments_stay_whole(layers, d, int8, n_kv, seqs, one, more):
    limit = one if layers == 1 else more
    for pages in (limit, limit + 1):
        a = KVArena(layers, 2 * n_kv, n_kv, d, 1024, 16, 256)
        s = [a.new_seq() for _ in range(seqs)]
        a.begin_step_host_only(s, [16 * pages - 1] * seqs)
        a.begin_step_host_only(s, [1] * seqs)
        pl = a.debug_decode_choice(0, int8, 4 if int8 and d <= 128 else 6, 296 if int8 and d <= 128 else 148)
        assert (pl["n_ctas"] == seqs * n_kv) == (pages == limit) and pl["n_ctas"] >= seqs * n_kv


@pytest.mark.skipif(torch.cuda.is_available(), reason="checks the behaviour on a machine without a GPU")
def test_compute_fails_loudly_without_a_gpu():
    a = arena()
    s = a.new_seq()
    lib = _lib.load()
    hs = (C.c_void_p * 1)(s._h)
    nt = (C.c_int64 * 1)(1)
    rc = lib.cbkv_begin_step(a._h, hs, nt, None, 1, None)
    assert rc == -5 and b"no CPU path" in lib.cbkv_last_error()
    assert s.seq_len() == 0  # nothing advanced
    assert lib.cbkv_attention(a._h, 0, None, None, None, None, 1.0, 0, None) == -6  # no step begun


def test_empty_step_changes_nothing():
    a = KVArena(2, 8, 2, 64, 64, num_pages=8)
    s = a.new_seq()
    a.begin_step_host_only([s], [20])
    free = a.num_free_pages()
    a.begin_step_host_only([], [])
    assert s.seq_len() == 20 and s.pages_used() == 2 and a.num_free_pages() == free


@pytest.mark.parametrize("lens,new,window,tokens,tile,kv_tile,sms,max_parts", [
    ([33], [2], 0, 32, 16, 128, 148, 64), ([1], [1], 0, 32, 16, 128, 148, 64), ([32000], [5], 0, 32, 16, 128, 148, 64),
    ([600, 6000, 128, 2500], [5] * 4, 0, 32, 16, 128, 148, 64), ([0, 4000, 127, 129], [512, 1, 1, 1], 0, 32, 16, 128, 148, 64),
    ([4608] * 2, [512] * 2, 0, 64, 32, 128, 148, 4), ([7000] * 8, [512] * 8, 0, 64, 32, 128, 148, 64),
    ([4500, 900], [512, 17], 1024, 64, 64, 64, 148, 64), ([4500, 900], [512, 17], 1024, 64, 64, 64, 148, 1),
    ([40000], [1000], 17, 64, 64, 64, 3, 64), ([5000] * 3, [300, 1, 1], 0, 128, 64, 128, 0, 64)])
def test_tile_plan_covers_every_kv_tile_once(lens, new, window, tokens, tile, kv_tile, sms, max_parts):
    # every (sequence, kv head, block of query tokens) exactly once, its slices gapless, in order and not empty, its
    # slots and its ticket its own
    a = KVArena(1, 28, 4, 128, 45000, 16, 20000)
    seqs = [a.new_seq() for _ in lens]
    for s_, n in zip(seqs, lens):
        if n:
            a.begin_step_host_only([s_], [n])
    a.begin_step_host_only(seqs, new)
    pl = a.debug_tile_plan(window, tokens, tile, kv_tile, sms, max_parts)
    want = {}
    for b, (pos, n) in enumerate(zip(lens, new)):
        for qt in range(-(-n // tokens)):
            first, last = pos + qt * tokens, pos + min((qt + 1) * tokens, n) - 1
            pages = last // 16 - (max(0, first - window + 1) if window else 0) // 16 + 1
            for h in range(4):
                want[b, h, qt] = -(-pages * 16 // kv_tile)
    got, slots, tickets = {}, set(), set()
    for b, h, qt, t0, t1, pn, base, cut in pl["tiles"].tolist():
        part, parts = pn & 0xffff, pn >> 16
        assert t1 > t0 and 1 <= parts <= max(1, max_parts)
        got.setdefault((b, h, qt), []).append((part, t0, t1))
        if parts == 1:
            assert base == cut == -1
        else:
            assert 0 <= base + part < pl["n_slots"] and base + part not in slots and 0 <= cut < pl["n_cut"]
            slots.add(base + part)
            tickets.add((cut, b, h, qt))
    assert len(tickets) == len({t[0] for t in tickets}) == pl["n_cut"] and len(slots) == pl["n_slots"]
    assert set(got) == set(want)
    for key, sl in got.items():
        sl.sort()
        assert [p for p, _, _ in sl] == list(range(len(sl)))
        assert sl[0][1] == 0 and sl[-1][2] == want[key] and all(x[2] == y[1] for x, y in zip(sl, sl[1:]))
    if max_parts == 1 or sms == 0:
        assert pl["n_cut"] == 0


@pytest.mark.parametrize("sms", [2, 7, 148])
def test_tile_plans_never_need_more_slots_than_the_buffers_have(sms):
    # the partial-result buffers are allocated once, for 4 slices per SM and half as many cut items
    a = KVArena(1, 28, 4, 128, 45000, 16, 60000)
    seqs = [a.new_seq() for _ in range(40)]
    for i, s_ in enumerate(seqs):
        a.begin_step_host_only([s_], [100 + 23 * i * i])
    for n in (1, 2, 9, 40):
        for new in ([5] * n, [1] * (n - 1) + [700]):
            a.begin_step_host_only(seqs[40 - n:], new)
            for window in (0, 1024):
                for tokens, tile, kv_tile in ((32, 16, 128), (16, 16, 128), (64, 64, 64)):
                    pl = a.debug_tile_plan(window, tokens, tile, kv_tile, sms)
                    assert pl["n_slots"] <= 4 * sms and pl["n_cut"] <= 2 * sms


@pytest.mark.parametrize("n_q,n_kv,d,n_seqs,new,lo,hi,kernel,most", [
    (32, 8, 128, 64, 3, 40, 100, 1, 0), (8, 4, 256, 64, 3, 40, 60, 1, 0), (8, 4, 256, 64, 3, 100, 1000, 2, 800), (32, 8, 128, 32, 3, 100, 1000, 3, 512),
    (28, 4, 128, 64, 5, 100, 3000, 3, 800), (32, 8, 128, 8, 5, 512, 6144, 3, 1496), (32, 8, 128, 1, 512, 512, 512, 6, 800)])
def test_a_chunk_kernel_is_chosen_without_modelling_every_launch(n_q, n_kv, d, n_seqs, new, lo, hi, kernel, most):
    # CTAs run through the launch model, which the host does in front of a step's first launch: none where the mma.sync
    # kernel is below what any plan could reach, and no more than the plan of one kernel takes when every candidate of its
    # cut is run (1536, 512, 2084, 1816, 2088, 1496 and 1392; 1024, 768, 1158, 1162, 1426, 928 and 848 more for pairs)
    lens = [int(lo + (i + 1) * 0.618 % 1 * (hi - lo)) for i in range(n_seqs)]
    a = KVArena(1, n_q, n_kv, d, 8192, 16, 16384)
    seqs = [a.new_seq() for _ in lens]
    a.begin_step_host_only(seqs, lens)
    a.begin_step_host_only(seqs, [new] * n_seqs)
    got = a.debug_chunk_choice()
    assert got["kernel"] == kernel and got["modelled"] <= most
    assert (got["n_ctas"] > 0) == (kernel != 1)


@pytest.mark.parametrize("sms", [2, 7, 148])
@pytest.mark.parametrize("n_q,n_kv,d", [(28, 4, 128), (8, 4, 256)])
def test_pairs_of_sms_never_need_more_slots_or_tickets_than_the_buffers_have(n_q, n_kv, d, sms):
    # the partial-result buffers: 4 slots per SM, of 256 rows at head_dim 128 and of 128 at head_dim 256, half as many
    # tickets; an item of a pair takes 256 rows a slot and a ticket for each of its two tiles
    a = KVArena(1, n_q, n_kv, d, 45000, 16, 60000)
    seqs = [a.new_seq() for _ in range(40)]
    for i, s_ in enumerate(seqs):
        a.begin_step_host_only([s_], [100 + 23 * i * i])
    for n in (1, 2, 9, 40):
        for new in ([5] * n, [1] * (n - 1) + [700], [512] * n):
            a.begin_step_host_only(seqs[40 - n:], new)
            for window in (0, 1024):
                pl = a.debug_chunk_choice(window, 6, sms)
                assert pl["kernel"] == 6 and pl["n_slots"] * (1 if d == 128 else 2) <= 4 * sms and 2 * pl["n_cut"] <= 2 * sms


@pytest.mark.parametrize("n_seqs,new,ctx,window,fastest", [
    (48, 2, 2048, 0, 2), (48, 5, 2048, 1024, 2), (48, 9, 8192, 0, 2), (16, 5, 8192, 0, 2), (16, 9, 512, 0, 2), (4, 2, 2048, 0, 2), (4, 9, 8192, 0, 2),
    (64, 5, 33, 0, 1), (1, 9, 8192, 0, 6), (1, 5, 2048, 1024, 6), (4, 9, 512, 0, 6), (1, 512, 512, 0, 6), (8, 512, 4096, 0, 6), (4, 512, 4096, 1024, 6)])
def test_head_dim_256_takes_the_kernel_that_was_measured_fastest(n_seqs, new, ctx, window, fastest):
    # 8 query and 4 kv heads on a B200, one tile / pairs / mma.sync, each row more than 5 % apart
    a = KVArena(1, 8, 4, 256, 16384, 16, 32768)
    seqs = [a.new_seq() for _ in range(n_seqs)]
    a.begin_step_host_only(seqs, [ctx] * n_seqs)
    a.begin_step_host_only(seqs, [new] * n_seqs)
    assert a.debug_chunk_choice(window)["kernel"] == fastest


@pytest.mark.parametrize("ctx,new,kernel", [
    ([1024, 1024], [333, 333], 3), ([2378, 921, 4276, 1655, 641, 2975, 1152, 5349], [5] * 8, 3), ([512], [512], 6), ([512], [100], 6)])
def test_head_dim_128_takes_pairs_only_where_they_are_faster(ctx, new, kernel):
    # 28 query and 4 kv heads on a B200, two tiles / pairs: 35 / 43 us, 29 / 32 a layer, and pairs faster in the other two
    a = KVArena(1, 28, 4, 128, 16384, 16, 32768)
    seqs = [a.new_seq() for _ in ctx]
    a.begin_step_host_only(seqs, ctx)
    a.begin_step_host_only(seqs, new)
    assert a.debug_chunk_choice()["kernel"] == kernel
