"""Compression where a tile is short: the warp that holds a segment's end takes
the masked path and the others the whole-block one, so segments are made to
end in every warp of a tile, inside, at and just past a block; float32,
float64 and both fastmodes, byte for byte against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,mode", [(8, 2), (16, 1), (32, 1), (32, 2), (64, 2), (256, 1), (256, 2)])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_segment_ends(szp, port, dtype, L, mode):
    import torch
    from szp_gb300.workloads import walk64
    rng = np.random.default_rng(L + mode)
    tile = 8192  # values of a tile at every blockSize
    for w in range(9):
        for past in (0, 1, 2, L // 2, L, L + 1):
            n = tile + w * 1024 + past
            x = walk64(n, rng)
            eb = float(np.float32(10.0 ** rng.uniform(-6, -2)))
            if dtype == "f32":
                x = x.astype(np.float32)
                want = port.compress(x, eb, L, 1, mode)
                cap = szp.max_stream_bytes(n, L, 1, mode)
                f = szp.compress_dev
            else:
                want = port.compress_d(x, eb, L, 1, mode)
                cap = szp.max_stream_bytes_f64(n, L, 1, mode)
                f = szp.compress_dev_f64
            d_x = torch.from_numpy(x).cuda()
            d_s = torch.zeros(cap, dtype=torch.uint8, device="cuda")
            size = f(d_x.data_ptr(), n, d_s.data_ptr(), cap, szp.ABS, eb, 0.0, L, 1, mode)
            assert d_s[:size].cpu().numpy().tobytes() == want, (n, eb)
