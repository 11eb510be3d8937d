"""Readback of normal forms on both sides of the size from which each subtree of
a net gets a warp of its own: sorted trees, one-sided lists (a split finds
nothing to share) and a batch that mixes sizes, against the oracle's texts."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))


def _list(n):
    t = "*"
    for i in range(n):
        t = f"({i % 9} {t})"
    return f"@main = {t}\n"


@pytest.mark.gpu
@pytest.mark.parametrize("shape,size", [("sort", d) for d in (1, 6, 9, 10, 11, 13)] + [("list", n) for n in (30, 500, 511, 3000)])
def test_gathered_text(shape, size):
    import hvm64
    import workloads as W
    from oracle import oracle
    text = W.bitonic(size, 3) if shape == "sort" else _list(size)
    want, _, _ = oracle.run_book(text)
    net = hvm64.Net(hvm64.Book.from_str(text), 512 << 20)
    net.boot("main")
    net.normal(hvm64.Tuning(timeout_ms=20000))
    assert net.readback() == want


@pytest.mark.gpu
def test_gathered_batch_of_mixed_sizes():
    import hvm64
    import workloads as W
    from oracle import oracle
    entries = [("sort", d, j) for j, d in enumerate((3, 11, 2, 12, 8, 10, 1, 9))] + [("sum", 5, 8)]
    text = W.batch_book(entries)
    batch = hvm64.Batch(hvm64.Book.from_str(text), [f"main_{j}" for _, _, j in entries], 1 << 30)
    batch.normal(hvm64.PERSISTENT, hvm64.Tuning(timeout_ms=20000))
    for i, (_, _, j) in enumerate(entries):
        assert batch.readback(i) == oracle.run_book(text, entry=f"main_{j}")[0]
