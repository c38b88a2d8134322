"""fastmode2 compression quantizes the values of its blocks and nothing else: a
block has one value fewer to pack than its lanes have places, and what lies
in shared memory after the last block of a tile (here the values of an
earlier field, all out of range) must not raise the notice of a clean field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [3e38, float("nan")])
@pytest.mark.parametrize("L", [8, 64, 256])
def test_clean_field_has_no_notice(szp, port, L, bad):
    import torch
    from szp_gb300.workloads import walk
    tile = 8192  # values of a tile at every blockSize
    n = 1000 * tile + 3 * 1024  # full tiles, and one that ends with a warp's share
    x = walk(n, np.random.default_rng(L))
    eb = float(np.float32(1e-3))
    want = port.compress(x, eb, L, 1, 2)
    d_x = torch.from_numpy(x).cuda()
    cap = szp.max_stream_bytes(n, L, 1, 2)
    d_s = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    # one float past a 16-byte boundary: a tile's last value then lies where the
    # clean field's tiles have the word after their last
    d_bad = torch.full((n + 1,), bad, dtype=torch.float32, device="cuda")
    for _ in range(3):
        szp.compress_dev(d_bad.data_ptr() + 4, n, d_s.data_ptr(), cap, szp.ABS, eb, 0.0, L, 1, 2)
        assert szp.last_notices() == 1
        size = szp.compress_dev(d_x.data_ptr(), n, d_s.data_ptr(), cap, szp.ABS, eb, 0.0, L, 1, 2)
        assert szp.last_notices() == 0
        assert d_s[:size].cpu().numpy().tobytes() == want
