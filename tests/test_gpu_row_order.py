"""GPU tier: the row encoder's items wait for those before them, and CUDA does not promise that
CTAs start in the order of their index.  An item that has waited too long leaves its place and
the publisher encodes it again: with the roles turned round (each item starts before everything
it waits for, the publisher last), and with items that leave at once or after a few polls while
the publisher is at work, the images are those of the usual order."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import to_dev

pytestmark = pytest.mark.gpu

P = ctypes.c_void_p


def _encode(lc, x, codec, bs, fit, wait, reversed_):
    import torch

    L, s, n = lc.lib(), x.element_size(), x.numel()
    cap = L.leco_max_payload_bytes(codec, s, n, bs)
    wsb = L.leco_encode_workspace_bytes(codec, s, n, bs, fit)
    nb = (n + bs - 1) // bs
    pay = torch.full((cap,), 0x5A, dtype=torch.uint8, device=x.device)
    off = torch.full((nb + 1,), -1, dtype=torch.int64, device=x.device)
    ws = torch.full((wsb,), 0xC3, dtype=torch.uint8, device=x.device)
    rc = L.leco_test_encode_order(codec, s, P(x.data_ptr()), n, bs, fit, P(pay.data_ptr()), cap, P(off.data_ptr()),
                                  P(ws.data_ptr()), wsb, wait, reversed_, P(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, L.leco_last_error()
    left = ws.cpu().numpy()[(nb * 8 + 255) // 256 * 256:].view(np.uint32)[1:3]
    lc.check()
    return pay, off, left


def _values(n, s, rng):
    if s == 8:
        return np.uint64(1 << 44) + np.cumsum(rng.integers(0, 1 << 18, n, dtype=np.uint64))
    return (np.arange(n, dtype=np.uint64) * 11 + rng.integers(0, 1 << 14, n, dtype=np.uint64)).astype(np.uint32)


# several blocks an item, one, and CTAs of 3, 8, 9 and 16 warps; waves: more CTAs than the GPU holds
CASES = [(8, 0, 1000, 400, False), (8, 0, 4096, 2000, True), (4, 1, 4096, 3500, True), (8, 2, 2048, 3000, True),
         (4, 3, 9000, 1500, True), (8, 1, 3000, 2500, True), (4, 0, 16384, 900, True), (8, 3, 8192, 300, False),
         (4, 2, 40, 50_000, True)]


@pytest.mark.parametrize("s,codec,bs,blocks,waves", CASES)
@pytest.mark.parametrize("wait,reversed_", [(256, 1), (1, 0), (20, 0), (0, 0)])
def test_any_order_gives_the_same_images(lc, dev, s, codec, bs, blocks, waves, wait, reversed_):
    import torch

    rng = np.random.default_rng(bs + blocks)
    x = to_dev(_values(bs * blocks - bs // 3, s, rng), dev)
    want = lc.encode(x, codec, bs, lc.FIT_REFERENCE)
    pay, off, left = _encode(lc, x, codec, bs, lc.FIT_REFERENCE, wait, reversed_)
    assert torch.equal(off, want.offsets)
    assert torch.equal(pay[: want.nbytes], want.payload[: want.nbytes])
    assert left[0] == left[1]  # every item that wanted to leave has gone on or is on the list
    if reversed_ and waves:  # those that start first wait for others that cannot start
        assert left[0] > 0
    if wait == 0:
        assert left[0] == 0
    lc.check()


def test_publisher_wait_runs_out(lc, dev):
    """The publisher waiting for an item's total gives up after its poll limit and reports it;
    what had been published before stays, the rest is not touched, and the context keeps working."""
    words = (ctypes.c_uint64 * 4)()
    assert lc.lib().leco_test_rows_wait(2000, words) == -5
    lc.check()  # the error word was read and cleared
    assert list(words) == [(2 << 62) | 48, 0, 0, 0]
    x = to_dev(np.arange(50_000, dtype=np.uint64) * 3, dev)
    col = lc.encode(x, lc.LINEAR, 1000)
    assert col.decode().equal(x)
    lc.check()
