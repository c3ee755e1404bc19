"""The native side of the Python calls: what it takes, what it leaves to the general path, and that both answer alike."""
import os
import subprocess
import sys

import pytest
import torch

from combsengine_b200 import CbkvError, KVArena, PagedKVCache, RotaryEmbedding, attention_rope
from combsengine_b200.kv import CacheConfig

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

STEPS = """
import ctypes as C
from combsengine_b200 import _lib
n = _lib.native()
I64, VP = C.c_int64, C.c_void_p
seen = []
def begin(arena, seqs, news, pos, m, stream):
    seen.append((arena, seqs[:m], news[:m], pos[:m] if pos else None, stream))
    return 7 if m == 3 else 0
def popn(seq, k, out):
    out[0] = min(k, 5)
    return 0
keep = [C.CFUNCTYPE(C.c_int32, VP, C.POINTER(VP), C.POINTER(I64), C.POINTER(I64), C.c_int32, VP)(begin),
        C.CFUNCTYPE(C.c_int32, VP, I64, C.POINTER(I64))(popn)]
n.bind(1, 1, *(C.cast(f, VP).value for f in keep))

class Stream:
    cuda_stream = 99
class Seq:
    def __init__(self, h): self._h = h
class Meddler:  # its attribute's getter changes a list of the call
    def __init__(self, *lists): self.lists = lists
    @property
    def _h(self):
        for l in self.lists: l.clear()
        return 5
a, b, st = Seq(11), Seq(12), Stream()

assert n.begin_step(1, [a, b], [3, 4], None, st) == (0, 7)
assert n.begin_step(1, [a, b], [3, 4], [8, 9], st) == (0, 7)
assert n.begin_step(1, [], [], None, st) == (0, 0)
assert n.begin_step(1, [a, a, b], [1, 1, 1], None, st) == (7, 3)  # the library's refusal comes back as its code
assert seen == [(1, [11, 12], [3, 4], None, 99), (1, [11, 12], [3, 4], [8, 9], 99), (1, [], [], None, 99), (1, [11, 11, 12], [1, 1, 1], None, 99)]
for args in [(1, (a, b), [3, 4], None, st), (1, [a, b], (3, 4), None, st), (1, [a, b], [3], None, st), (1, [a, b], [3, 4], [1], st),
             (1, [a, b], [3.0, 4], None, st), (1, [a, b], [3, 2 ** 70], None, st), (None, [a, b], [3, 4], None, st), (1, [a, object()], [3, 4], None, st),
             (1, [a, Seq(None)], [3, 4], None, st), (1, [a, b], [3, 4], None, 99), (1, [a, b], [3, 4], None)]:
    assert n.begin_step(*args) == n.SLOW, args
news, pos = [3] * 200, [0] * 200
for args in [(news,), (pos,)]:
    x, y = [3] * 200, [0] * 200
    seqs = [a] * 199 + [b]
    seqs[0] = Meddler(x if args[0] is news else y)
    assert n.begin_step(1, seqs, x, y, st) == n.SLOW
seqs = [a] * 200
seqs[0] = Meddler(seqs)
assert n.begin_step(1, seqs, news, pos, st) == n.SLOW
assert len(seen) == 4

assert n.popn(11, 3) == (0, 3) and n.popn(11, 9) == (0, 5)
for args in [(None, 3), (11, 3.0), (11, 2 ** 70), (11,)]:
    assert n.popn(*args) == n.SLOW, args
import torch
t = torch.zeros(8, dtype=torch.float16)
assert n.attention(1, 0, t, t, t, None, 1.0, None, st, 0, 8, 8) == n.SLOW  # not on a GPU
assert n.attention_rope(1, 0, 1, 0, t, t, t, None, 1.0, None, st, 0, 8, 8) == n.SLOW
"""


def test_steps_and_rollbacks_without_a_gpu():
    # in a process of its own: the module is bound to functions that write down what reaches the library
    r = subprocess.run([sys.executable, "-c", STEPS], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr


@pytest.mark.gpu
def test_both_paths_take_and_refuse_the_same_calls():
    answers = []
    for native in (True, False):
        g = KVArena(1, 8, 2, 64, 256, 16, 32)
        if not native:
            g._native = None
        gen = torch.Generator(device="cuda").manual_seed(1)
        rand = lambda n: torch.randn(n, generator=gen, device="cuda", dtype=torch.float16)
        s, other, got = g.new_seq(), torch.cuda.Stream(), []
        rope = RotaryEmbedding(g, 10000.0, 256)
        q, k, v = rand(20 * 8 * 64), rand(20 * 2 * 64), rand(20 * 2 * 64)

        def call(f, *args, **kw):
            try:
                r = f(*args, **kw)
                got.append(r.clone() if isinstance(r, torch.Tensor) else r)
                return r
            except (CbkvError, TypeError, ValueError, AttributeError) as e:
                got.append((type(e).__name__, getattr(e, "msg", "")))

        call(g.attention, 0, q, k, v, 0.1)                      # no step yet
        call(g.begin_step, (s,), (20,), (0,))                   # tuples
        call(g.begin_step, [s], [20], [5])                      # a position that is not the sequence's
        for name, x in (("bf16", q.bfloat16()), ("short", q[:-64]), ("strided", rand(2 * 20 * 8 * 64)[::2]), ("host", q.cpu()), ("list", [1.0])):
            call(g.attention, 0, x, k, v, 0.1)
        out = torch.empty_like(q)
        assert call(g.attention, 0, q, k, v, 0.1, out=out) is out
        assert call(g.attention, 0, q.view(20, 8, 64), k, v, 0.1).shape == (20, 8, 64)
        call(g.attention, 1, q, k, v, 0.1)                      # no such layer
        call(g.attention, 0, q, k, v, 0.1, window=1)            # no such window
        call(g.attention, 0, q, k, v, 0.1, window=4)
        call(attention_rope, g, 0, rope, q, k, v, 0.1)
        call(attention_rope, g, 0, rope, q, k[:-64], v, 0.1)
        other.wait_stream(torch.cuda.current_stream())
        call(g.attention, 0, q, k, v, 0.1, out=out, stream=other)
        torch.cuda.synchronize()
        got.append(out.clone())
        call(s.popn, 7)
        call(s.popn, 700)
        call(g.begin_step, [s], [300])                          # more than there are pages
        got.append((g.step_tokens, s.seq_len(), g.device_status()))
        rope.close()
        g.close()
        call(s.popn, 1)
        answers.append(got)
        cache = PagedKVCache(1, CacheConfig(256), 8, 2, 64)
        if not native:
            cache.arena._native = None
        q4, k4 = q.view(1, 8, 20, 64), k.view(1, 2, 20, 64)
        got.append(cache.attention_opts(0, q4, k4, v.view(1, 2, 20, 64), 0, 0.1))
        got.append(cache.attention_opts(0, q4.transpose(1, 2).contiguous().transpose(1, 2), k4, v.view(1, 2, 20, 64), 20, 0.1))
    assert len(answers[0]) == len(answers[1])
    for x, y in zip(*answers):
        assert torch.equal(x, y) and x.shape == y.shape if isinstance(x, torch.Tensor) else x == y, (x, y)
