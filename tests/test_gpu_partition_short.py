"""GPU tier: the device partitioner on both sides of the rule that gives columns of many short
coarse blocks a thread per block, against the host partitioner.  Segment starts are whole
numbers: bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs,blocks", [(1, 749), (1, 750), (2, 1499), (2, 1501), (3, 20_000), (16, 11_999), (16, 12_000),
                                       (33, 24_750), (80, 60_000), (81, 60_750)])
@pytest.mark.parametrize("kind", ["regimes", "noise"])
def test_short_blocks_match_host(lc, dev, bs, blocks, kind):
    import torch
    from leco_b200 import workloads

    n = bs * blocks + (bs - 1) // 2  # a last block that is not whole
    if kind == "regimes":
        x = workloads.regime_switching_u64(n, seed=bs, mean_regime=500.0)
    else:
        x = torch.randint(0, 1 << 62, (n,), generator=torch.Generator().manual_seed(bs))
    want = lc.varlen_partition(x.numpy().view(np.uint64), n // bs, 12)
    got = lc.varlen_partition_device(x.to(dev), n // bs, 12)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), want)
    lc.check()
