"""Work shared from a single waiting redex on: nearly every slot a warp fills
holds redexes that the selection of the same step has just put back on its
stack.  A redex lost, doubled or torn on the way would change the normal form
or the counts, which equal the oracle's on every run."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [1, 0])
@pytest.mark.parametrize("kind,size", [("sort", 4), ("sort", 9), ("sum", 11), ("church", 3)])
def test_redexes_put_back_and_shared_at_once(kind, size, blocks):
    import hvm64
    import workloads as W
    from oracle import oracle
    text = {"sort": W.bitonic, "sum": W.tree_sum}[kind](size, 3) if kind != "church" else W.church_big((3, 2, size))
    want, want_rw, _ = oracle.run_book(text)
    net = hvm64.Net(hvm64.Book.from_str(text), 512 << 20)
    net.boot("main")
    for _ in range(5):
        rw = net.normal(hvm64.Tuning(timeout_ms=20000, donate_min=1, blocks_per_sm=blocks))
        assert net.readback() == want
        assert rw.as_dict() == want_rw
    assert net.stats()["donated"] > 0
