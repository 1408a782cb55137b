"""GPU tier: a kernel's opt-in to more than 48 KB of shared memory belongs to the kernel, so a
call with small blocks must not take it away from one with large blocks."""
import numpy as np
import pytest

from gpu_helpers import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big,small", [((0, 4096), (1, 4096)), ((3, 4096), (0, 256)), ((3, 16384), (1, 16384))])
def test_older_batch_encodes_after_a_smaller_one(lc, dev, big, small):
    """Batch A (LeCo or degree-2 u64 items: the fit's tables beside the values), then batch B
    (smaller items); A still encodes, by a launch and by a graph's first capture."""
    import torch

    rng = np.random.default_rng(big[0] * 100 + small[0])
    x = np.cumsum(rng.integers(0, 5000, 60_000, dtype=np.uint64)) + np.uint64(1 << 45)
    xd = to_dev(x, dev)
    a = lc.Batch([(xd, *big)])
    b = lc.Batch([(xd, *small)])
    for batch, (codec, bs) in ((a, big), (b, small)):
        one = lc.encode(xd, codec, bs, lc.FIT_REFERENCE)
        for run in (batch.encode, lambda: batch.run_graph(3)):
            c = batch.cols[0]
            c.payload.zero_()
            run()
            assert torch.equal(c.offsets, one.offsets)
            assert torch.equal(c.payload[: one.nbytes], one.payload[: one.nbytes])
    lc.check()
