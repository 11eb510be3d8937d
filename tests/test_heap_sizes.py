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


@pytest.mark.gpu
@pytest.mark.parametrize("kind,depth,nets,mb", [("sum", 6, 64, 3), ("sum", 10, 64, 30), ("sort", 7, 32, 12)])
def test_plain_batches_in_small_heaps(kind, depth, nets, mb):
    """One net a launch, every net's nodes kept: the lanes of every launch must
    not cost the batch a chunk each."""
    import hvm64
    import workloads as W
    from oracle import oracle
    text = W.batch_book([(kind, depth, j) for j in range(nets)])
    names = [f"main_{j}" for j in range(nets)]
    batch = hvm64.Batch(hvm64.Book.from_str(text), names, mb << 20)
    batch.normal(hvm64.PLAIN, hvm64.Tuning(timeout_ms=20000))
    for i in (0, 1, nets - 1):
        want, want_rw, _ = oracle.run_book(text, entry=names[i])
        assert batch.readback(i) == want
        assert batch.rwts[i].as_dict() == want_rw
