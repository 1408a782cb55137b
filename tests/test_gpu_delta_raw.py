"""GPU tier: raw blocks of a u32 Delta column in the staged decoder (written from the staged
image) -- block sizes on both sides of the staging buffer and of the warp kernel's, outputs
that do not start on 32 bytes, raw and packed blocks side by side -- and the same column's sum.
Whole numbers: bit-exact."""
import numpy as np
import pytest

from gpu_helpers import to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", [512, 513, 1000, 2049, 4096, 4160, 4200, 8192])
@pytest.mark.parametrize("mixed", [False, True])
def test_raw_blocks(lc, dev, bs, mixed):
    import torch

    rng = np.random.default_rng(bs)
    n = bs * 1030 + 5  # the staged decoder takes columns of 1024 blocks and more
    x = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    if mixed:  # every third block packed
        i = np.arange(n)
        x = np.where(i // bs % 3 == 1, (i * 7 % 100_000).astype(np.uint32), x)
    col = lc.encode(to_dev(x, dev), lc.DELTA, bs)
    buf = torch.zeros(n + 16, dtype=torch.int32, device=dev)
    for shift in (0, 1, 3, 4):
        out = buf[shift:shift + n]
        buf.fill_(-1)
        assert np.array_equal(to_np(col.decode(out=out), 4), x), (bs, shift)
        assert int((buf[:shift] != -1).sum()) == 0 and int((buf[shift + n:] != -1).sum()) == 0
    assert col.sum() == int(x.astype(np.uint64).sum()) & (2**64 - 1)
    first, count = bs - 3, 2 * bs + 7
    assert np.array_equal(to_np(col.decode_range(first, count), 4), x[first:first + count])
    lc.check()
