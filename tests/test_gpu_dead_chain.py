"""A stream whose header chain breaks: a block's bit count is set to a value that
no block has, at the first, an inner and the last block of a segment and around
a chunk's and a super-chunk's start.  The blocks behind it must not be counted
(other lanes and CTAs found their headers), so every such stream is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _headers(s, n, L, T, mode):
    """Offsets of every block's bit-count byte, by segment."""
    size = lambda m, b: 1 if b == 0 else 1 + (m + 7) // 8 + (b >> 3) * m + ((b & 7) * m + 7) // 8
    off = np.frombuffer(s[4:4 + 8 * T], "<u8")
    out = []
    for t in range(T):
        lo, hi = t * (n // T), n if t == T - 1 else (t + 1) * (n // T)
        p, e, at = 4 + 8 * T + int(off[t]) + (4 if mode == 1 else 0), lo + (1 if mode == 1 else 0), []
        while e < hi:
            m = min(L, hi - e) - (mode == 2)
            at.append(p + (4 if mode == 2 else 0))
            p = at[-1] + size(m, s[at[-1]]) if m else at[-1] + 1
            e += L
        out.append((at, 4 + 8 * T + int(off[t])))
    return out


@pytest.mark.parametrize("L,mode", [(8, 1), (32, 1), (32, 2), (64, 1), (256, 2)])
def test_broken_chain_is_refused(szp, port, L, mode):
    import torch
    from szp_gb300.workloads import walk
    n, T = 150_001, 3
    x = walk(n, np.random.default_rng(L))
    s = port.compress(x, float(np.float32(2e-4 * np.ptp(x))), L, T, mode)
    out = torch.zeros(n, device="cuda")
    for at, start in _headers(s, n, L, T, mode):
        pick = {0, 1, len(at) // 2, len(at) - 2, len(at) - 1}
        for edge in (1024, 2048, 16384):  # the blocks on both sides of a chunk's or super-chunk's start
            i = int(np.searchsorted(np.array(at) - start, edge))
            pick |= {i - 1, i, i + 1}
        for i in sorted(k for k in pick if 0 <= k < len(at)):
            for b in (34, 255):
                bad = bytearray(s)
                bad[at[i]] = b
                if mode == 2 and L > 1 and i == len(at) - 1 and (n // T) % L == 1:
                    continue  # a one-value block has no bit count that is read
                buf = torch.frombuffer(bad, dtype=torch.uint8).cuda()
                szp.decompress_dev(buf.data_ptr(), len(bad), n, out.data_ptr(), L, T, mode)
                assert szp.sync_status() == szp.ECORRUPT, (L, mode, i, b)
    buf = torch.frombuffer(bytearray(s), dtype=torch.uint8).cuda()  # and the GPU is as it was
    szp.decompress_dev(buf.data_ptr(), len(s), n, out.data_ptr(), L, T, mode)
    assert szp.sync_status() == 0
    assert np.array_equal(out.cpu().numpy().view(np.uint32), port.decompress(s, n, L, T, mode).view(np.uint32))
