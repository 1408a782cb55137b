"""GPU tier: the row encoder's CTA sizes -- blocks of 65 and more rows have a CTA of their own,
of as many warps as the rows need (3, 5, 6, 9 to 14) or of the next power of two -- at the
edges of each size, and columns of more items than one step of the offsets' publisher with any
of them.  Byte work: bit-exact against the oracle."""
import numpy as np
import pytest

from gpu_helpers import expected_gpu_column, mask_delta_last_fields, to_dev, to_np

pytestmark = pytest.mark.gpu

EDGES = [2048, 2049, 3072, 3073, 4096, 4097, 5120, 5121, 6144, 6145, 7168, 7169, 8192, 8193, 9216, 9217, 10_241, 11_265, 12_288,
         12_289, 13_312, 13_313, 14_336, 14_337, 16_383]


def _keys(n, s, rng):
    if s == 8:  # sums above 2^53, as the reference's chain sees them
        return np.uint64(1 << 44) + np.cumsum(rng.integers(0, 1 << 18, n, dtype=np.uint64))
    return (np.arange(n, dtype=np.uint64) * 11 + rng.integers(0, 500, n, dtype=np.uint64)).astype(np.uint32)


@pytest.mark.parametrize("s", [4, 8])
@pytest.mark.parametrize("bs", EDGES)
def test_images_at_the_edges(lc, orc, dev, s, bs):
    rng = np.random.default_rng(3 * bs + s)
    x = _keys(3 * bs + bs // 3, s, rng)
    xd = to_dev(x, dev)
    for codec in range(4):
        epay, eoff, _ = expected_gpu_column(orc, codec, x, bs)
        col = lc.encode(xd, codec, bs, lc.FIT_REFERENCE)
        pay, off = col.to_host()
        if codec == 2:
            pay, epay = (mask_delta_last_fields(p, o, s, len(x), bs) for p, o in ((pay, off), (epay, eoff)))
        assert np.array_equal(off, eoff) and np.array_equal(pay, epay), codec
        assert np.array_equal(to_np(col.decode(), s), x), codec
        if codec in (0, 3):  # the exact moments' form of the fit
            assert np.array_equal(to_np(lc.encode(xd, codec, bs, lc.FIT_EXACT).decode(), s), x), codec
    lc.check()


@pytest.mark.parametrize("bs,blocks", [(32, 17_000), (1024, 1300), (2049, 900), (4097, 700), (9000, 1200), (14_000, 600)])
def test_many_items(lc, orc, dev, bs, blocks):
    """Every block's offset, over several steps of the publisher."""
    rng = np.random.default_rng(bs)
    n = bs * (blocks - 1) + 1
    x = rng.integers(0, 1 << 20, n, dtype=np.uint64).astype(np.uint32) >> rng.integers(0, 20, blocks).astype(np.uint32).repeat(bs)[:n]
    col = lc.encode(to_dev(x, dev), lc.FOR, bs)
    pay, off = col.to_host()
    epay, eoff, _ = expected_gpu_column(orc, 1, x, bs)
    assert np.array_equal(off, eoff) and np.array_equal(pay, epay)
    lc.check()


@pytest.mark.parametrize("codec,bs,blocks", [(0, 9000, 4095), (0, 9000, 4096), (0, 5000, 6143), (0, 5000, 6144), (3, 5000, 2559),
                                             (3, 5000, 2560), (3, 12_300, 2560)])
def test_fits_inside_and_before(lc, dev, codec, bs, blocks):
    """Both sides of the block counts from which the fit kernels run before the encoder leave the
    images of a short column, which always takes the fits inside."""
    import torch

    g = torch.Generator(device=dev).manual_seed(bs + blocks)
    n = bs * blocks - bs // 2
    x = (torch.arange(n, device=dev, dtype=torch.int64) * 70_001 + (1 << 41)
         + torch.randint(0, 5000, (n,), generator=g, device=dev, dtype=torch.int64))
    col = lc.encode(x, codec, bs, lc.FIT_REFERENCE)
    k = 300
    for at in (0, blocks - k):
        short = lc.encode(x[at * bs:min(n, (at + k) * bs)], codec, bs, lc.FIT_REFERENCE)
        base = int(col.offsets[at].item())
        assert torch.equal(col.offsets[at:at + k + 1] - base, short.offsets)
        assert torch.equal(col.payload[base:base + short.nbytes], short.payload[: short.nbytes])
    assert torch.equal(col.decode(), x)
    lc.check()
