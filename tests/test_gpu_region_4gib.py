"""Decoding a segment whose blocks end within a super-chunk of 4 GiB, the most
that a segment's 32-bit offsets reach: the ends of its last super-chunk and of
its last, short block are formed without passing 2^32.  The stream is made on
the GPU: every block has 32 bits a value and the same signs and magnitudes, so
that the values alternate between the seed and the seed plus one delta."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# blockSize 8 and 256 take the one-kernel decode, 24 the per-block passes; with m
# values in the last block the regions end 4, 22, 82 and 1039 bytes below 4 GiB,
# and a last block taken for a whole one ends past it for (8, 3) and (24, 3)
@pytest.mark.parametrize("L,m", [(8, 3), (8, 7), (24, 3), (256, 5)])
def test_region_of_4_gib(szp, port, L, m):
    import torch
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GB of device memory")
    size = lambda k: 1 + (k + 7) // 8 + 4 * k  # bytes of a block of k values of 32 bits
    block = np.array([32] + [0x55] * (L // 8) + [0x40] * (4 * L), np.uint8)
    short = np.array([32] + [0x55] * ((m + 7) // 8) + [0x40] * (4 * m), np.uint8)
    assert block.size == size(L) and short.size == size(m)
    seed, delta = 5, 0x40404040

    def stream(blocks):
        head = np.frombuffer(np.array([1.0], ">f4").tobytes() + bytes(8) + np.array([seed], "<i4").tobytes(), np.uint8)
        s = torch.empty(head.size + blocks * block.size + short.size, dtype=torch.uint8, device="cuda")
        s[:head.size] = torch.from_numpy(head.copy()).cuda()
        s[head.size:head.size + blocks * block.size].view(blocks, block.size)[:] = torch.from_numpy(block).cuda()
        s[-short.size:] = torch.from_numpy(short).cuda()
        return s, 1 + blocks * L + m

    s, n = stream(3)  # the oracle agrees on what the pattern decodes to
    want = port.decompress(s.cpu().numpy().tobytes(), n, L, 1, 1)
    assert np.array_equal(want[0::2], np.full((n + 1) // 2, np.float32(seed)))
    assert np.array_equal(want[1::2], np.full(n // 2, np.float32(seed + delta)))

    blocks = ((1 << 32) - 1 - short.size) // block.size
    s, n = stream(blocks)
    assert (1 << 32) - 1200 < s.numel() - 16 < 1 << 32
    y = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")
    szp.decompress_dev(s.data_ptr(), s.numel(), n, y.data_ptr(), L, 1, 1)
    assert szp.sync_status() == 0, szp.last_error()
    assert bool((y[0::2] == float(np.float32(seed))).all())
    assert bool((y[1::2] == float(np.float32(seed + delta))).all())
