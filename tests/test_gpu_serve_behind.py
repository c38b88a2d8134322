"""A server with far more requests than its lanes take: the decoder runs fewer
CTAs there, and every result is the one that a server with nothing waiting, and
one with a single lane, gives for the same request."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_batch,lanes", [(2, 3), (1, 2), (4, 1), (64, 3)])
def test_server_behind(szp, port, max_batch, lanes):
    import torch
    from szp_gb300.workloads import walk
    from test_gpu_serve import _copy
    T = 4
    rng = np.random.default_rng(max_batch)
    fields = []
    for n in (1, 4099, 70_000, 900_001):
        x = walk(n, rng)
        eb = float(np.float32(2e-4 * (np.ptp(x) + 1e-3)))
        s = port.compress(x, eb, 32, T, 1)
        fields.append((torch.from_numpy(x).cuda(), n, eb, torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda(), s,
                       port.decompress(s, n, 32, T, 1)))
    torch.cuda.synchronize()
    srv = szp.Server(2 << 30, max_batch=max_batch, lanes=lanes, segments=T)
    reqs = []
    for k in range(120):
        x, n, eb, d_s, s, y = fields[int(rng.integers(0, len(fields)))]
        if k % 3 == 0:
            reqs.append((s, dict(op=szp.BATCH_COMPRESS, input=x.data_ptr(), nbEle=n, errBoundMode=szp.ABS, absErrBound=eb)))
        else:
            reqs.append((y.tobytes(), dict(op=szp.BATCH_DECOMPRESS, input=d_s.data_ptr(), input_bytes=len(s), nbEle=n)))
    for rid, (want, r) in zip(srv.submit([r for _, r in reqs]), reqs):
        res = srv.wait(rid)
        assert res["status"] == 0
        got = torch.empty(len(want), dtype=torch.uint8, device="cuda")
        _copy(got.data_ptr(), res["output"], len(want))
        assert got.cpu().numpy().tobytes() == want
        srv.release(rid)
    srv.close()
