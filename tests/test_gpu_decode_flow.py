"""decode_flow where it can go wrong, against the oracle bit for bit: every
blockSize it takes and both fastmodes, every 32-byte phase of the output and
16-byte phase of the stream, super-chunks of one and of several chunks, runs of
empty blocks longer than a chunk and than the block list, every bit count, and
segments that end inside, at and just past a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(kind, n, rng):
    from szp_gb300.workloads import walk, bitcount_sweep
    if kind == "walk":
        return walk(n, rng)
    if kind == "empty":  # one value now and then in a constant field
        x = np.zeros(n, np.float32)
        x[rng.integers(0, n, 1 + n // 40000)] = 1.0
        return x
    if kind == "runs":  # runs of empty blocks of many lengths between noisy stretches
        x = walk(n, rng)
        p = 0
        while p < n:
            p += int(rng.integers(1, 3000))
            q = p + int(2 ** rng.uniform(3, 16))
            x[p:q] = x[p - 1] if p < n else 0.0
            p = q
        return x
    return np.tile(bitcount_sweep(rng), n // 2000 + 1)[:n]  # bit counts 0..33 (eb = 1)


@pytest.mark.parametrize("kind", ["walk", "empty", "runs", "bits"])
@pytest.mark.parametrize("L,mode", [(8, 1), (16, 2), (32, 1), (32, 2), (64, 1), (128, 2), (256, 1)])
def test_decode_flow(szp, port, kind, L, mode):
    import torch
    rng = np.random.default_rng(L * 10 + mode)
    for it, (n, T) in enumerate([(L + 1, 1), (L + 2, 1), (33 * L, 5), (20_011, 3), (700_000 + L, 16), (2_000_003, 7)]):
        x = _field(kind, n, rng)
        eb = 1.0 if kind == "bits" else float(np.float32(2e-4 * (float(np.ptp(x)) + 1e-3)))
        s = port.compress(x, eb, L, T, mode)
        want = port.decompress(s, n, L, T, mode).view(np.uint32)
        for off in range(it, it + 8, 3):  # output and stream phases
            d_s = torch.zeros(len(s) + 16, dtype=torch.uint8, device="cuda")
            d_s[off:off + len(s)] = torch.frombuffer(bytearray(s), dtype=torch.uint8).cuda()
            d_y = torch.full((n + 16,), 7.0, dtype=torch.float32, device="cuda")
            szp.decompress_dev(d_s.data_ptr() + off, len(s), n, d_y.data_ptr() + 4 * off, L, T, mode)
            assert szp.sync_status() == 0, szp.last_error()
            y = d_y.cpu().numpy()
            assert np.array_equal(y[off:off + n].view(np.uint32), want), (n, T, off)
            assert np.all(y[:off] == 7.0) and np.all(y[off + n:] == 7.0)


def test_decode_flow_turns(szp, port):
    """Segments of very different sizes, and more of them than take turns."""
    rng = np.random.default_rng(5)
    for n, T in ((3_000_000, 4), (1_000_000, 600)):
        x = _field("walk", n, rng)
        x[: n // 2] = 0.0
        s = port.compress(x, 1e-4, 32, T, 1)
        szp.set_segments(T)
        y = szp.szp_decompress(s, n, 32, 1)
        szp.set_segments(0)
        assert np.array_equal(y.view(np.uint32), port.decompress(s, n, 32, T, 1).view(np.uint32)), (n, T)
