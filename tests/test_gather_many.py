"""Readback of runs with many nets: a few normal forms big enough for a warp
per subtree among thousands of small ones, and more big ones than get such a
split (each is then one warp's walk, as it is when the device has no memory for
the splits).  Texts equal the oracle's."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))


SMALL = "@small = (1 (2 (3 *)))\n"


def _sort(depth):
    import workloads as W
    return W.bitonic(depth, 3) + SMALL


def _check(src, names):
    import hvm64
    from oracle import oracle
    want = {n: oracle.run_book(src, entry=n)[0] for n in set(names)}
    batch = hvm64.Batch(hvm64.Book.from_str(src), names, 4 << 30)
    batch.normal(hvm64.PERSISTENT, hvm64.Tuning(timeout_ms=20000))
    for i, n in enumerate(names):
        assert batch.readback(i) == want[n], i


@pytest.mark.gpu
def test_a_few_big_normal_forms_among_thousands():
    names = ["small"] * 4200
    for i in (0, 17, 2100, 4199):
        names[i] = "main"
    _check(_sort(12), names)


@pytest.mark.gpu
@pytest.mark.parametrize("big", [512, 513])
def test_more_big_normal_forms_than_are_split(big):
    _check(_sort(11), ["main"] * big + ["small"] * 3)
