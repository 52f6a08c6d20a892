"""A program's layout (folded relations, shift schedule, trees) is made by its
first prove on a context and read by the later ones: every order in which
proves, verifications, refused calls and sessions share a context gives the
proof that a context of its own gives."""
import pytest

from loom_b200 import Context, LoomError, field as F, plonk, transcript

pytestmark = pytest.mark.gpu


def _case(sizes, seed):
    compiled, wit = plonk.build_mixed(sizes, seed=seed)
    return compiled, [F.to_mont(w) for w in wit]


def _own(compiled, mont, q):
    ctx = Context(0)
    try:
        return ctx.prove(compiled.words, mont, q)
    finally:
        ctx.close()


@pytest.mark.parametrize("first", ["prove", "verify", "refused", "session"])
def test_shared_context_equals_own_context(first):
    a, wa = _case([6, 4, 7, 5], 3)
    b, wb = _case([4, 4], 4)
    want = _own(a, wa, 9)
    ctx = Context(0)
    if first == "verify":
        ctx.verify(a.words, want, 9)
    elif first == "refused":
        with pytest.raises(LoomError):
            ctx.prove(a.words, wa, 0)
        with pytest.raises(LoomError):
            ctx.prove(a.words[:-1], wa, 9)
    elif first == "session":
        ctx.session(a.words, wa, 9).release()  # begun, never driven
    assert ctx.prove(a.words, wa, 9) == want
    assert ctx.prove(b.words, wb, 5) == _own(b, wb, 5)
    assert ctx.prove(a.words, wa, 9) == want
    assert ctx.prove(a.words, wa, 3) == _own(a, wa, 3)  # other query count, same program
    with pytest.raises(LoomError):
        ctx.prove(a.words, wa, 0)
    ctx.verify(a.words, want, 9)
    ctx.close()


def test_sessions_of_one_program_interleaved_and_evicted():
    a, wa = _case([5, 6], 7)
    want = _own(a, wa, 4)
    ctx = Context(0)
    s, t = ctx.session(a.words, wa, 4), ctx.session(a.words, wa, 4)
    for k in range(20):  # more programs than a context keeps
        c, wc = plonk.build(1 + k % 7, 1 << (4 + k // 7), seed=100 + k)
        ctx.prove(c.words, [F.to_mont(w) for w in wc], 2)
    for x in (s, t):
        assert transcript.drive(x, a.modules, a.n_rounds, 4, None) == want
        x.release()
    assert ctx.prove(a.words, wa, 4) == want
    ctx.close()
