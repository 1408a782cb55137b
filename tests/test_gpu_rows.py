"""GPU tier: the row encoder (one thread per row of 32 values) where it can go wrong --
block sizes around its group sizes (8, 16, 32, 64, 128, 256, 512 rows), partial rows, source
pointers that are not 16-byte aligned, widths up to 64 bits -- and its parallel form of the
reference's sequential sums.  Everything is integer or byte work: bit-exact against the
oracle."""
import numpy as np
import pytest

from gpu_helpers import expected_gpu_column, mask_delta_last_fields, to_dev, to_np

pytestmark = pytest.mark.gpu


def _family(name, n, s, rng):
    top = 2 ** (8 * s) - 1
    if name == "noise":  # wide rows, raw blocks
        return rng.integers(0, top, n, dtype=np.uint64, endpoint=True)
    if name == "steep":  # sums far above 2^53: chains, binade passes
        return (rng.uniform(0, top / 4.0 / max(n, 1)) * np.arange(n)).astype(np.uint64) + rng.integers(0, 4096, n, dtype=np.uint64)
    if name == "level":  # large and nearly constant
        return np.uint64(top) - rng.integers(0, 9, n, dtype=np.uint64)
    if name == "jump":  # several binades passed inside one row
        return np.where(np.arange(n) < n // 3, np.uint64(5), np.uint64(top // 3)) + rng.integers(0, 3, n, dtype=np.uint64)
    if name == "powers":
        return np.uint64(1) << rng.integers(0, 8 * s, n, dtype=np.uint64)
    if name == "nanoseconds":  # predictions above 2^51
        return np.uint64(top // 11) + np.cumsum(rng.integers(0, 2_000_000 if s == 8 else 20, n, dtype=np.uint64))
    return np.full(n, top // 5, np.uint64)  # constant


@pytest.mark.parametrize("s", [4, 8])
@pytest.mark.parametrize("bs", [1, 2, 31, 32, 33, 255, 257, 513, 1000, 1025, 2048, 2049, 4095, 4096, 4097, 8193, 16384])
def test_images_match_oracle(lc, orc, dev, s, bs):
    rng = np.random.default_rng(100 * bs + s)
    dt = np.uint64 if s == 8 else np.uint32
    for name in ("noise", "steep", "level", "jump", "powers", "nanoseconds", "constant"):
        n = min(3 * bs + int(rng.integers(0, bs + 1)), 40_000)
        x = _family(name, n + 1, s, rng).astype(dt)
        xd = to_dev(x, dev)
        for codec in range(4):
            for first in (0, 1):  # 1: a source that starts on one value, not on 16 bytes
                v = x[first:first + n]
                col = lc.encode(xd[first:first + n], codec, bs, lc.FIT_REFERENCE)
                pay, off = col.to_host()
                epay, eoff, _ = expected_gpu_column(orc, codec, v, bs)
                if codec == 2:
                    pay, epay = (mask_delta_last_fields(p, o, s, n, bs) for p, o in ((pay, off), (epay, eoff)))
                assert np.array_equal(off, eoff) and np.array_equal(pay, epay), (name, codec, s, bs, first)
                assert np.array_equal(to_np(col.decode(), s), v), (name, codec, s, bs, first)
    lc.check()


@pytest.mark.parametrize("n", [4096 * 8191, 4096 * 8192 + 5])
def test_large_column_fit_paths_agree(lc, dev, n):
    """The fit inside the row encoder (fewer than 8192 blocks) and the fit kernels (from
    there on) leave the same images: the first blocks of a column are those of a short one."""
    import torch

    g = torch.Generator(device=dev).manual_seed(n)
    x = (torch.arange(n, device=dev, dtype=torch.int64) * 70_001 + (1 << 41)
         + torch.randint(0, 5000, (n,), generator=g, device=dev, dtype=torch.int64))
    col = lc.encode(x, lc.LINEAR, 4096, lc.FIT_REFERENCE)
    short = lc.encode(x[:4096 * 500], lc.LINEAR, 4096, lc.FIT_REFERENCE)
    assert torch.equal(col.offsets[:501], short.offsets)
    assert torch.equal(col.payload[: short.nbytes], short.payload[: short.nbytes])
    assert torch.equal(col.decode(), x)
    lc.check()


@pytest.mark.parametrize("bs", [256, 1000, 4096, 8192, 16384])
def test_batch_items_match_single_columns(lc, dev, bs):
    """Encoder items of several blocks (256 threads) and of one 512-row block in one batch."""
    import torch

    rng = np.random.default_rng(bs)
    specs, cols = [], []
    for k in range(12):
        s, codec = (4, 8)[k % 2], k % 4
        n = int(rng.integers(1, 5 * bs))
        x = _family(("steep", "noise", "nanoseconds")[k % 3], n, s, rng).astype(np.uint64 if s == 8 else np.uint32)
        cols.append((to_dev(x, dev), codec))
        specs.append((cols[-1][0], codec, bs))
    specs.append((cols[0][0], 0, 16384))
    cols.append((cols[0][0], 0))
    b = lc.Batch(specs)
    b.encode()
    b.decode()
    for (v, codec), c in zip(cols, b.cols):
        one = lc.encode(v, codec, c.block_size, lc.FIT_REFERENCE)
        assert torch.equal(one.offsets, c.offsets), (codec, bs)
        assert torch.equal(one.payload[: one.nbytes], c.payload[: one.nbytes]), (codec, bs)
        assert torch.equal(one.dir, c.dir) and torch.equal(c.out, v), (codec, bs)
    lc.check()
