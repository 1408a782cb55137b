"""GPU tier: the row encoder's ways past its 32-bit residuals -- blocks in which every warp of
rows, some warps, single rows or single values do not fit them, and neighbours in one warp that
differ -- for the codecs with a model.  Byte work: bit-exact against the oracle."""
import numpy as np
import pytest

from gpu_helpers import expected_gpu_column, to_dev, to_np

pytestmark = pytest.mark.gpu


def _column(kind, n, s, rng):
    i = np.arange(n, dtype=np.uint64)
    smooth = i * np.uint64(7) + np.uint64(10**6) + rng.integers(0, 9, n, dtype=np.uint64)
    wide = rng.integers(0, 1 << (41 if s == 8 else 32), n, dtype=np.uint64)
    if kind == "all":
        return wide
    if kind == "warps":  # every other 1024 values
        return np.where((i >> np.uint64(10)) & np.uint64(1), wide, smooth)
    if kind == "rows":  # every third row of 32
        return np.where((i >> np.uint64(5)) % np.uint64(3) == 1, wide, smooth)
    if kind == "late":  # a row's first values fit, its last do not
        return np.where(i & np.uint64(31) > 28, wide, smooth)
    if kind == "early":  # its first value alone does not
        return np.where(i & np.uint64(31) == 0, wide, smooth)
    x = smooth.copy()  # one value of the column
    x[n // 2] = np.uint64(2 ** (8 * s - 1) + 5)
    return x


@pytest.mark.parametrize("s", [4, 8])
@pytest.mark.parametrize("bs", [32, 100, 256, 700, 1500, 2049, 4096, 5000, 9000])
def test_wide_blocks(lc, orc, dev, s, bs):
    rng = np.random.default_rng(10 * bs + s)
    dt = np.uint64 if s == 8 else np.uint32
    n = min(4 * bs + bs // 3, 24_000)
    for kind in ("all", "warps", "rows", "late", "early", "one"):
        x = _column(kind, n, s, rng).astype(dt)
        for codec in (0, 3):
            col = lc.encode(to_dev(x, dev), codec, bs, lc.FIT_REFERENCE)
            pay, off = col.to_host()
            epay, eoff, _ = expected_gpu_column(orc, codec, x, bs)
            assert np.array_equal(off, eoff) and np.array_equal(pay, epay), (kind, codec)
            assert np.array_equal(to_np(col.decode(), s), x), (kind, codec)
    lc.check()
