"""GPU tier: the order in which the row encoder's items wait for one another rests on a ticket,
not on the order in which CUDA starts the CTAs of a grid."""
import numpy as np
import pytest

from gpu_helpers import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s,codec,n,bs,items", [(8, 0, 100_000, 1000, 25), (4, 1, 5 * 4096 + 1, 4096, 6), (8, 2, 65_536, 8, 512)])
def test_every_role_is_a_ticket(lc, dev, s, codec, n, bs, items):
    """The workspace is one status word per block, then the ticket.  After an encode it has been
    taken once per item and once for the publisher, and every item's status word holds the
    inclusive prefix of the sizes, which is its last block's end."""
    import torch

    x = to_dev(np.arange(n, dtype=np.uint64 if s == 8 else np.uint32) * 3, dev)
    nb = (n + bs - 1) // bs
    ws = torch.empty(int(lc.lib().leco_encode_workspace_bytes(codec, s, n, bs, lc.FIT_REFERENCE)), dtype=torch.uint8, device=dev)
    col = lc.encode(x, codec, bs, lc.FIT_REFERENCE, workspace=ws)
    words = ws.cpu().numpy().view(np.uint64)
    assert int(words[(nb * 8 + 255) // 256 * 32] & np.uint64(0xFFFFFFFF)) == items + 1
    off = col.offsets.cpu().numpy().view(np.uint64)
    per = -(-nb // items)
    assert np.array_equal(words[:items], np.uint64(2 << 62) | off[np.minimum(np.arange(1, items + 1) * per, nb)])
    assert torch.equal(col.decode(), x)
    lc.check()


@pytest.mark.parametrize("part", [0, 1])
def test_waits_run_out(lc, dev, part):
    """The publisher waiting for an item's total and an item waiting for its prefix both give up
    after their poll limit and report it; what had been published before stays, the rest is not
    touched, and the context keeps working."""
    import ctypes

    words = (ctypes.c_uint64 * 4)()
    assert lc.lib().leco_test_rows_wait(2000, part, words) == -5
    lc.check()  # the error word was read and cleared
    assert list(words) == ([(2 << 62) | 48, 0, 0, 0] if part == 0 else [0, 0, 0, 2**64 - 1])
    x = to_dev(np.arange(50_000, dtype=np.uint64) * 3, dev)
    col = lc.encode(x, lc.LINEAR, 1000)
    assert col.decode().equal(x)
    lc.check()
