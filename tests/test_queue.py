"""The device redex queue at the edges of its ring: capacities from the
smallest (16 slots: every push takes the compare-and-swap path and the ring
wraps many times) to ones whose pushes take tickets, work shared from a single
waiting redex on, several runs on one handle (each run's tickets start above
the last one's, over the words the last one left) and runs of different
capacities in turn.  Normal forms and counts equal the oracle's."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))


@pytest.mark.gpu
@pytest.mark.parametrize("donate_min", [0, 1, 33])
@pytest.mark.parametrize("qlog2", [4, 6, 13, 17])
def test_queue_capacities(qlog2, donate_min):
    import hvm64
    import workloads as W
    from oracle import oracle
    text = W.bitonic(8, 5)
    want, want_rw, _ = oracle.run_book(text)
    net = hvm64.Net(hvm64.Book.from_str(text), 512 << 20)
    net.boot("main")
    for q in (qlog2, qlog2, 18, qlog2):
        rw = net.normal(hvm64.Tuning(timeout_ms=20000, queue_slots_log2=q, donate_min=donate_min))
        assert net.readback() == want
        assert rw.as_dict() == want_rw


@pytest.mark.gpu
def test_queue_graph_replays():
    import hvm64
    import workloads as W
    from oracle import oracle
    entries = [("sum", 3 + j % 5, j) if j % 2 else ("sort", 2 + j % 6, j) for j in range(37)]
    text = W.batch_book(entries)
    book = hvm64.Book.from_str(text)
    batch = hvm64.Batch(book, [f"main_{j}" for _, _, j in entries], 1 << 30)
    want = [oracle.run_book(text, entry=f"main_{j}")[:2] for _, _, j in entries]
    for flags in (hvm64.TUNE_GRAPH, hvm64.TUNE_GRAPH, 0, hvm64.TUNE_GRAPH):
        batch.normal(hvm64.PERSISTENT, hvm64.Tuning(timeout_ms=20000, flags=flags))
        for i, (t, rw) in enumerate(want):
            assert batch.readback(i) == t
            assert batch.rwts[i].as_dict() == rw
