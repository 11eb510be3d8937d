"""The instruction kinds on ports of nodes a call makes itself (I_CALL, I_FCTR,
I_FFLINK, I_FCONST) against the oracle, over the shapes the encoder can meet:
constants that reach a constructor, a variable, an operator or a switch; trees
in a call's argument; links of two own ports (of one node, of two, across
redexes); redexes between two constructors (wires of an own node); and the same
shapes under an argument, where they may be wires of consumed nodes.  CPU: the
emulation of the device runtime.  GPU: the library."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))
sys.path.insert(0, HERE)

LIB = "@id = (a a)\n@fst = (a (* a))\n@swap = ((a b) (b a))\n@sw = (?((5 (x x)) r) r)\n"
SHAPES = {
    "call_tree": "@main = r & @fst ~ (7 (8 r))",
    "call_nested": "@main = r & @id ~ ((1 (2 *)) r)",
    "own_pair_one_node": "@main = r & @id ~ ((a a) r)",
    "own_pair_two_nodes": "@main = r & @id ~ ((a b) q) & @id ~ ((b a) s) & @id ~ (q (s r))",
    "const_var": "@main = (a a) & 3 ~ a2 & @id ~ (a2 b) & @id ~ (b c) & @id ~ (c *)",
    "const_num_ctr": "@main = (a b) & 9 ~ (a b)",
    "const_era_ctr": "@main = (a b) & * ~ (a b)",
    "const_op": "@main = a & 4 ~ $([+3] a)",
    "const_op_ref": "@main = a & 4 ~ $([*] $(b a)) & @id ~ (6 b)",
    "const_switch": "@main = a & 0 ~ ?((1 (x x)) a)",
    "const_switch_pos": "@main = a & 3 ~ ?((1 (x x)) a)",
    "own_op": "@main = r & @id ~ (a r) & @id ~ (5 $([+2] a))",
    "own_switch": "@main = r & @id ~ (2 ?((1 (x x)) r))",
    "ref_switch": "@main = r & @sw ~ (3 r)",
    "two_ctrs": "@main = r & (1 r) ~ (a a)",
    "two_ctrs_labels": "@main = (p q) & (p q) ~ #2{1 2}",
    "two_ctrs_deep": "@main = r & ((1 2) r) ~ ((a b) (b a))",
    "argument": "@f = ((a (b c)) (c (b a)))\n@main = r & @f ~ ((1 (2 3)) r)",
    "argument_era": "@f = ((a (* c)) (c a))\n@main = r & @f ~ (* r)",
    "argument_dup": "@f = (#1{a b} (a b))\n@main = r & @f ~ ((1 (x x)) r)",
    "argument_self": "@f = ((a a) b)\n& @id ~ (7 b)\n@main = r & @f ~ ((x x) r)",
    "argument_mixed": "@f = ((a b) c)\n& @swap ~ ((a 4) (d e))\n& @fst ~ (e (d (b c)))\n@main = r & @f ~ ((1 2) (r *))",
}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_shapes_on_the_emulation(name):
    import test_emu
    from oracle import oracle
    src = LIB + SHAPES[name] + "\n"
    want, want_rw, _ = oracle.run_book(src)
    for threads in (1, 4):
        text, rw = test_emu.emu_run(src, threads=threads, heap=1 << 20)
        assert text == want
        assert rw == want_rw


@pytest.mark.gpu
def test_shapes_on_the_gpu():
    import hvm64
    from oracle import oracle
    for name in sorted(SHAPES):
        src = LIB + SHAPES[name] + "\n"
        want, want_rw, _ = oracle.run_book(src)
        net = hvm64.Net(hvm64.Book.from_str(src), 256 << 20)
        net.boot("main")
        rw = net.normal(hvm64.Tuning(timeout_ms=20000))
        assert (name, net.readback(), rw.as_dict()) == (name, want, want_rw)
