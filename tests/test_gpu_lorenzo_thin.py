"""The Lorenzo variant on thin fields, byte for byte and bit for bit: one row or
one plane (passes that leave work out), and lines below, at and past the 16
values that the inverse sums load at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 4096), (1, 1, 4099), (7, 1, 4096), (15, 1, 333), (1, 16, 1000), (2, 17, 999),
                                  (16, 2, 1000), (17, 3, 1001), (31, 33, 64), (1, 2, 40_001), (40_001, 1, 1)])
def test_thin_fields(szp, port, dims):
    import torch
    rng = np.random.default_rng(sum(dims))
    n = int(np.prod(dims))
    f = (np.cumsum(rng.standard_normal(n)) * 0.01).astype(np.float32)
    eb = float(np.float32(1e-4 * (np.ptp(f) + 1e-3)))
    want = port.lorenzo_compress(f, dims, eb, 3)
    y = port.lorenzo_decompress(want, dims, 3)
    cap = szp.lorenzo_max_stream_bytes(dims, 3)
    for off in (0, 1):  # 16-byte aligned, and not
        d_x = torch.zeros(n + 1, device="cuda")
        d_x[off:off + n] = torch.from_numpy(f).cuda()
        d_s = torch.zeros(cap, dtype=torch.uint8, device="cuda")
        size = szp.lorenzo_compress_dev(d_x.data_ptr() + 4 * off, dims, d_s.data_ptr(), cap, szp.ABS, eb, 0.0, 3)
        assert szp.last_notices() == 0
        assert d_s[:size].cpu().numpy().tobytes() == want
        d_y = torch.full((n + 2,), 7.0, device="cuda")
        szp.lorenzo_decompress_dev(d_s.data_ptr(), size, dims, d_y.data_ptr() + 4 * off, 3)
        out = d_y.cpu().numpy()
        assert np.array_equal(out[off:off + n].view(np.uint32), np.asarray(y, np.float32).view(np.uint32))
        assert np.all(out[:off] == 7.0) and np.all(out[off + n:] == 7.0)
