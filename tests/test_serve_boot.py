"""Requests whose boot leaves many redexes: counts on both sides of a queue
slot (32) and of the warp's stack (512), in one burst, several times over, so
that many warps boot at once.  Every result equals the oracle's."""
import os
import sys
import time

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, os.path.join(ROOT, "hvm-64_b200"))

SIZES = (0, 1, 2, 31, 32, 33, 64, 65, 200, 511, 512, 513)


def _serve(sizes, tuning, rounds):
    import hvm64
    from oracle import oracle
    src = "@id = (a a)\n" + "".join(f"@b{n} = (r {n})\n& @id ~ (7 r)\n" + "& @id ~ (1 *)\n" * n for n in sizes)
    want = {n: oracle.run_book(src, entry=f"b{n}")[:2] for n in sizes}
    sv = hvm64.Server(hvm64.Book.from_str(src), slots=3 * len(sizes), out_pairs=1 << 10, heap_bytes=1 << 30, tuning=tuning)
    try:
        for _ in range(rounds):
            owner = {sv.submit(f"b{n}"): n for n in sizes for _ in range(3)}
            end = time.time() + 20
            while owner and time.time() < end:
                for t in sv.poll():
                    text, rw, _ = sv.result(t)
                    n = owner.pop(t)
                    assert (n, text, rw.as_dict()) == (n, *want[n])
            assert not owner
    finally:
        sv.close()


@pytest.mark.gpu
def test_boots_of_many_redexes():
    import hvm64
    _serve(SIZES, hvm64.Tuning(timeout_ms=60000), 20)


@pytest.mark.gpu
def test_boots_that_find_the_queue_full():
    """A queue of 16 slots and boots of more redexes than it holds slots, or
    than the warp's stack holds: what the queue does not take is reduced by
    the warp that booted the request."""
    import hvm64
    _serve((1, 33, 513, 600, 1100), hvm64.Tuning(timeout_ms=60000, queue_slots_log2=4), 20)
