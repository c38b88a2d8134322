"""The decode's ticket map over segment counts at the edges of its rules: one
to three segments, turns up to 512 segments, a thread each above; and
super-chunks of few chunks that share the room for notes, from fields whose
blocks take 1.3 to 8 bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("T", [1, 3, 4, 511, 512, 513, 1500, 5000])
def test_segment_counts(szp, port, T, mode):
    import torch
    from szp_gb300.workloads import walk
    rng = np.random.default_rng(T)
    for n, rel in ((700_003, 1e-3), (3 * T + 1, 1e-4)):
        x = walk(n, rng)
        eb = float(np.float32(rel * (float(np.ptp(x)) + 1e-3)))
        s = port.compress(x, eb, 32, T, mode)
        want = port.decompress(s, n, 32, T, mode)
        buf = torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda()
        out = torch.full((n,), float("nan"), device="cuda")
        szp.decompress_dev(buf.data_ptr(), len(s), n, out.data_ptr(), 32, T, mode)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32)), (n, rel)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("rel", [3e-2, 1e-2, 3e-3, 1e-3, 3e-4])
def test_dense_blocks(szp, port, rel, mode):
    import torch
    from szp_gb300.workloads import walk
    n = 6_000_011
    x = walk(n, np.random.default_rng(int(1e5 * rel)))
    eb = float(np.float32(rel * float(np.ptp(x))))
    for T in (1, 16):
        s = port.compress(x, eb, 32, T, mode)
        want = port.decompress(s, n, 32, T, mode)
        buf = torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda()
        out = torch.full((n,), float("nan"), device="cuda")
        szp.decompress_dev(buf.data_ptr(), len(s), n, out.data_ptr(), 32, T, mode)
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.asarray(want, np.float32).view(np.uint32)), T
