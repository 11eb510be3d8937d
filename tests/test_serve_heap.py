"""What a server's allocator may hold back, which its smallest heap and its node
budget follow from: 32 + 32 nodes a lane and 64 a warp."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [1, 4])
def test_smallest_heap_and_its_budget(blocks):
    import hvm64
    import torch
    warps = torch.cuda.get_device_properties(0).multi_processor_count * blocks * 2
    held = warps * (32 * 64 + 64)
    book = hvm64.Book.from_str("@main = x & 3 ~ $([*] $(5 x))\n")
    tuning = hvm64.Tuning(timeout_ms=60000, blocks_per_sm=blocks)
    with pytest.raises(hvm64.HvmError) as e:
        hvm64.Server(book, slots=4, out_pairs=64, heap_bytes=2 * held * 16, tuning=tuning)
    assert e.value.code == hvm64.ERR_BAD_INPUT
    sv = hvm64.Server(book, slots=4, out_pairs=64, heap_bytes=(2 * held + 1) * 16, tuning=tuning)
    try:
        assert sv.budget()["budget"] == held + 1
    finally:
        sv.close()
