"""Calls of Defs longer than the window of instructions a step stages, where
one call's node is matched by another call of the same step before its words
are filled by an instruction past the window (of the same lane, the next one or
the one after): the waiting lane must not keep the filling one from getting
there.  Normal forms and counts equal the oracle's.  CPU: the emulation of the
device runtime (a lane waits for a thread).  GPU: the library, where both calls
are lanes of one warp."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))
sys.path.insert(0, HERE)

# @f's node for its first argument, (u v), leaves through that argument at
# the call's second instruction; its words are filled by the last ones.
CALLS = ("& @f ~ (* z) & @f ~ (z *)", "& @f ~ (z *) & @f ~ (* z)")


def _book(fillers, calls, pairs=1, tail="(* *)"):
    f = f"@f = ((u v) {tail})\n" + "& @id ~ (1 *)\n" * fillers + "& @id ~ (u v)\n"
    main = " ".join(calls.replace("z", f"z{k}") for k in range(pairs))
    return f"@id = (a a)\n{f}@main = * {main}\n"


# 50, 65 and 128 instructions
LONG = [(f, c, p) for f in (14, 19, 40) for c in (0, 1) for p in (1, 16)]


@pytest.mark.parametrize("fillers,calls,pairs", LONG)
def test_long_defs_on_the_emulation(fillers, calls, pairs):
    import test_emu
    from oracle import oracle
    src = _book(fillers, CALLS[calls], pairs)
    want, want_rw, _ = oracle.run_book(src)
    text, rw = test_emu.emu_run(src, threads=8, heap=1 << 22)
    assert text == want
    assert rw == want_rw


@pytest.mark.gpu
@pytest.mark.parametrize("fillers,calls,pairs", LONG)
def test_long_defs_on_the_gpu(fillers, calls, pairs):
    import hvm64
    from oracle import oracle
    src = _book(fillers, CALLS[calls], pairs)
    want, want_rw, _ = oracle.run_book(src)
    net = hvm64.Net(hvm64.Book.from_str(src), 256 << 20)
    net.boot("main")
    rw = net.normal(hvm64.Tuning(timeout_ms=20000))
    assert net.readback() == want
    assert rw.as_dict() == want_rw


# 30, 32, 33 and 35 instructions: both sides of the staged window's end
EDGE = [(8, "*"), (8, "(* *)"), (9, "*"), (9, "(* *)")]


@pytest.mark.gpu
@pytest.mark.parametrize("fillers,tail", EDGE)
def test_defs_at_the_windows_end(fillers, tail):
    import hvm64
    from oracle import oracle
    for calls in CALLS:
        src = _book(fillers, calls, 16, tail)
        want, want_rw, _ = oracle.run_book(src)
        net = hvm64.Net(hvm64.Book.from_str(src), 256 << 20)
        net.boot("main")
        rw = net.normal(hvm64.Tuning(timeout_ms=20000))
        assert net.readback() == want
        assert rw.as_dict() == want_rw
