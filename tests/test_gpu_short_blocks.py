"""Decoding fields whose blocks take little more than a byte each: super-chunks
limited by their blocks and not by their bytes, chunks of an eighth of their size
and more for short blockSizes, and stretches (noisy, constant, alternating) where
the walking lanes have room for the notes and where they have not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(kind, n, rng):
    from szp_gb300.workloads import walk
    x = walk(n, rng)
    if kind == "modulated":  # slow and steep stretches
        i = np.arange(n)
        return (x * 0.05 + np.sin(2e-4 * i) * (1 + np.sin(7e-6 * i))).astype(np.float32)
    if kind == "patches":  # a third of constant stretches, and some where every other block is empty
        p = 0
        while p < n:
            q = p + int(rng.integers(20_000, 200_000))
            k = rng.integers(0, 3)
            if k == 0:
                x[p:q] = x[p]
            if k == 1:
                m = np.arange(p, min(q, n))
                x[m] = np.where((m // 40) % 2 == 0, x[p], x[m])
            p = q
    return x


@pytest.mark.parametrize("kind", ["walk", "modulated", "patches"])
@pytest.mark.parametrize("L,mode", [(8, 1), (8, 2), (16, 1), (16, 2), (32, 1), (64, 1), (128, 2), (256, 1)])
def test_short_blocks(szp, port, kind, L, mode):
    import torch
    n = 3_000_011
    x = _field(kind, n, np.random.default_rng(L + mode))
    for rel, T in ((0.3, 16), (0.03, 1), (0.01, 16), (3e-3, 3), (1e-3, 16), (2e-4, 1)):
        eb = float(np.float32(rel * float(np.ptp(x))))
        s = port.compress(x, eb, L, T, mode)
        want = port.decompress(s, n, L, T, mode)
        buf = torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda()
        out = torch.full((n,), float("nan"), device="cuda")
        szp.decompress_dev(buf.data_ptr(), len(s), n, out.data_ptr(), L, T, mode)
        assert szp.sync_status() == 0, szp.last_error()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32)), (rel, T)
