"""Nets in heaps not much larger than they need: work is shared out to every
warp of the device, which must not cost each of their lanes a full chunk of
fresh nodes."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,depth,mb", [("sum", 10, 3), ("sum", 14, 32), ("sum", 16, 96), ("sort", 5, 1),
                                           ("sort", 9, 16), ("sort", 11, 32)])
def test_nets_in_small_heaps(kind, depth, mb):
    import hvm64
    import workloads as W
    from oracle import oracle
    text = (W.tree_sum if kind == "sum" else W.bitonic)(depth, 1)
    want, want_rw, _ = oracle.run_book(text)
    net = hvm64.Net(hvm64.Book.from_str(text), mb << 20)
    net.boot("main")
    for _ in range(3):
        rw = net.normal(hvm64.Tuning(timeout_ms=20000))
        assert net.readback() == want
        assert rw.as_dict() == want_rw
