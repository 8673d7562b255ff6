"""A context made and run while the default stream is busy gives what it gives on an idle GPU: nothing of its set-up
may be left to the default stream, which its runs do not wait for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRODUCTS = ("clus", "xg", "zg", "cells", "tuple_off", "quality", "idv", "zv")


def test_busy_default_stream(conditions, events_pu50):
    import torch
    from pixeltrack import PixelChain, default_params
    blob, offs = events_pu50
    event = bytes(blob[offs[0]:offs[1]])

    def run():
        with PixelChain(conditions, default_params()) as chain:
            before = chain.sync()  # nothing has run yet: no warnings
            warn = chain.run_event(event)
            return before, warn, [chain.product(p).copy() for p in PRODUCTS]

    idle = run()
    stream = torch.cuda.default_stream()
    with torch.cuda.stream(stream):
        junk = torch.full((64 << 20,), 0x7F, dtype=torch.uint8, device="cuda")  # left in the allocator's memory
        torch.cuda._sleep(500_000_000)  # a quarter of a second
        junk.fill_(0x55)
    busy = run()
    torch.cuda.synchronize()
    assert idle[0] == busy[0] == 0 and idle[1] == busy[1]
    for name, a, b in zip(PRODUCTS, idle[2], busy[2]):
        assert np.array_equal(a, b), name
