"""GPU tier: the device partitioner's warp per coarse block (blocks of up to 8000 values) and
its thread per coarse block above that, against the host partitioner (which the CPU tier pins
to the reference), at block sizes around a warp's width, the lane / warp boundary of the pair
sizes (48 values) and the 8000-value limit, on values whose fit sums stay below 2^53, pass it
and start far above it.  Segment starts are whole numbers: bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(kind, n, rng):
    i = np.arange(n, dtype=np.uint64)
    if kind == "steps":
        return np.repeat(rng.integers(0, 1 << 40, n // 37 + 1, dtype=np.uint64), 37)[:n] + rng.integers(0, 9, n, dtype=np.uint64)
    if kind == "line":  # one long segment a block: pairs sized by the whole warp
        return np.uint64(1 << 43) + i * np.uint64(77_777) + rng.integers(0, 50, n, dtype=np.uint64)
    if kind == "curve":
        return (i * i) // np.uint64(7) + np.uint64(10**9) + rng.integers(0, 300, n, dtype=np.uint64)
    if kind == "high":  # near 2^63: 128-bit predictions, sums far above 2^53
        return np.uint64((1 << 63) - 1000) + i * np.uint64(3) + rng.integers(0, 4, n, dtype=np.uint64)
    return rng.integers(0, 2**64 - 1, n, dtype=np.uint64, endpoint=True)  # differences that wrap


@pytest.mark.parametrize("bs", [2, 31, 33, 48, 49, 65, 1000, 2000, 7999, 8000, 8001])
def test_matches_host(lc, dev, bs):
    import torch

    rng = np.random.default_rng(bs)
    for kind in ("steps", "line", "curve", "high", "noise"):
        for blocks, tail in ((3, 0), (2, 1), (5, bs // 2)):
            n = bs * blocks + tail
            coarse = max(1, n // bs)
            x = _values(kind, n, rng)
            for delta in (0, 12):
                want = lc.varlen_partition(x, coarse, delta)
                got = lc.varlen_partition_device(torch.from_numpy(x.view(np.int64)).to(dev), coarse, delta)
                assert np.array_equal(got.cpu().numpy().view(np.uint64), want), (kind, bs, n, delta)
    lc.check()
