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


@pytest.mark.parametrize("op", ["partition", "varlen", "legacy"])
def test_threads_with_different_block_sizes(lc, dev, op):
    """Two host threads, one with blocks that need the opt-in in full and one with smaller ones:
    every call of both succeeds."""
    import threading

    import torch

    rng = np.random.default_rng(7)
    x = np.cumsum(rng.integers(0, 5000, 64_000, dtype=np.uint64)) + np.uint64(1 << 40)
    xd, xs = to_dev(x, dev), to_dev((x & np.uint64(0xFFFFFFF)).astype(np.uint32), dev)
    sizes = {"partition": (8000, 4000), "varlen": (16_000, 6_400), "legacy": (16_000, 12_800)}[op]
    errors = []

    def work(bs):
        s = torch.cuda.Stream()
        try:
            with torch.cuda.stream(s):
                if op == "varlen":
                    starts = torch.arange(0, len(x), bs, device=dev, dtype=torch.int64)
                for _ in range(300):
                    if op == "partition":
                        lc.varlen_partition_device(xd[: 2 * bs], 2, 12)
                    elif op == "varlen":
                        lc.varlen_encode(xd, starts, max_segment_len=bs)
                    else:
                        lc.encode(xs, 5, bs)
            s.synchronize()
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append((bs, e))

    threads = [threading.Thread(target=work, args=(bs,)) for bs in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    lc.check()
