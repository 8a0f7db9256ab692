"""The pool of page-locked blocks: what a freed block waits for before it is handed out again."""
import threading
import time

import numpy as np
import pytest
import torch

import tatara_b200 as tb

pytestmark = pytest.mark.gpu

MB = 1 << 20  # every test uses a size class of its own, in which no other test leaves blocks


def _queue_copy(block, stream, value):
    """A copy from the block to the device behind a bounded delay, on a stream the library does not know."""
    block.array[:] = value
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)  # about 0.1 s
        return torch.from_numpy(block.array).to("cuda", non_blocking=True)


@pytest.mark.parametrize("other_thread", [False, True])
def test_a_freed_block_waits_for_copies_on_the_callers_own_stream(other_thread):
    torch.zeros(1, device="cuda")
    n = (21 + 2 * other_thread) * MB
    stream = torch.cuda.Stream()
    blocks = [tb.PinnedArray((n,), np.uint8) for _ in range(3)]
    addresses = {b.array.ctypes.data for b in blocks}
    got = [_queue_copy(b, stream, 7) for b in blocks]
    for b in blocks:
        if other_thread:
            t = threading.Thread(target=b.free)
            t.start()
            t.join()
        else:
            b.free()
    again = tb.PinnedArray((n,), np.uint8)  # all three still in use: the one freed first, behind the copies
    assert again.array.ctypes.data in addresses
    again.array[:] = 9
    stream.synchronize()
    assert all(bool((g == 7).all()) for g in got)


def test_an_idle_block_goes_first():
    """A loader that frees a batch behind a running step gets the block of an earlier batch, without waiting for the step."""
    torch.zeros(1, device="cuda")
    stream = torch.cuda.Stream()
    early, late = tb.PinnedArray((25 * MB,), np.uint8), tb.PinnedArray((25 * MB,), np.uint8)
    first = early.array.ctypes.data
    early.free()
    between = tb.PinnedArray((4096,), np.uint8)  # a later allocation: from here on the block waits for nothing new
    torch.cuda.synchronize()
    got = _queue_copy(late, stream, 7)
    late.free()
    t0 = time.perf_counter()
    block = tb.PinnedArray((25 * MB,), np.uint8)
    assert time.perf_counter() - t0 < 0.05 and not stream.query()
    assert block.array.ctypes.data == first
    stream.synchronize()
    assert bool((got == 7).all())
    between.free()
