"""Ticket pushes past the ring's first lap: 296 warps on a ring of 2^14 slots
take tickets (the rule asks for about 40 slots a warp), and a run that shares
more slots than that goes round it, each push waiting for the slot's previous
holder.  Normal forms and counts equal the oracle's."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))


@pytest.mark.gpu
def test_tickets_go_round_the_ring():
    import hvm64
    import workloads as W
    from oracle import oracle
    text = W.bitonic(12, 5)
    want, want_rw, _ = oracle.run_book(text)
    net = hvm64.Net(hvm64.Book.from_str(text), 512 << 20)
    net.boot("main")
    for _ in range(3):
        rw = net.normal(hvm64.Tuning(timeout_ms=20000, blocks_per_sm=1, queue_slots_log2=14, donate_min=1))
        assert net.readback() == want
        assert rw.as_dict() == want_rw
        assert net.stats()["donated"] > 2 << 14
