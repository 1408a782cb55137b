"""GPU tier: the kernels that take the reference's fits of a column of many blocks before its
encoder runs -- the ring of 16-byte copies (aligned values, blocks of whole 16 bytes) and the
tiled kernel (the rest), for LeCo u64 and degree-2 u32 and u64 -- at the block counts from which
they are used and one below.  The sums of the values leave 2^53 behind, so that the order of
the additions shows.  Byte work: every image, the short last block's too, against the oracle."""
import numpy as np
import pytest

from gpu_helpers import expected_gpu_column, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,codec,bs,shift", [
    (8, 0, 256, 0),  # ring
    (8, 0, 256, 1),  # tiled: values 8 bytes off
    (8, 0, 257, 0),  # tiled: blocks of an odd number of values
    (8, 0, 34, 0),   # ring, a tile of fewer than 32 values in every block
    (8, 3, 256, 0), (8, 3, 256, 1), (8, 3, 257, 0),
    (4, 3, 256, 0), (4, 3, 256, 1), (4, 3, 258, 0), (4, 3, 36, 0),
])
def test_images_match_oracle(lc, orc, dev, s, codec, bs, shift):
    rng = np.random.default_rng(1000 * codec + bs + shift)
    first = 8192 if codec == 0 else 5120
    for blocks, short in ((first - 1, 0), (first, 0), (first + 33, bs // 2 + 1), (first + 70, bs - 1)):
        n = bs * blocks - short
        if s == 8:
            x = np.uint64(1 << 52) + np.cumsum(rng.integers(0, 1 << 30, n, dtype=np.uint64))
        else:
            x = (np.uint64(1 << 31) + rng.integers(0, 1 << 30, n, dtype=np.uint64)).astype(np.uint32)
        buf = to_dev(np.concatenate([np.zeros(shift, x.dtype), x]), dev)
        col = lc.encode(buf[shift:], codec, bs, lc.FIT_REFERENCE)
        pay, off = col.to_host()
        epay, eoff, _ = expected_gpu_column(orc, codec, x, bs)
        assert np.array_equal(off, eoff) and np.array_equal(pay, epay), (blocks, short)
        assert np.array_equal(to_np(col.decode(), s), x)
    lc.check()
