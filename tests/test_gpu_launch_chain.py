"""Kernels launched behind the one before them (range -> compress, setup ->
decode) read what that one wrote, call after call without a host
synchronisation and in a captured graph, where the launches are ordinary."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _in_thread(fn):
    out = []

    def run():
        try:
            fn()
        except BaseException as e:  # noqa: BLE001 - handed to the caller below
            out.append(e)

    t = threading.Thread(target=run)
    t.start()
    t.join()
    if out:
        raise out[0]


@pytest.mark.parametrize("fm", [1, 2])
@pytest.mark.parametrize("n", [1, 33, 20011, 600000])
@pytest.mark.parametrize("graph", [False, True])
def test_calls_without_a_synchronisation(n, fm, graph):
    import torch

    import szp_gb300 as szp

    T, cap = 16, 8 * 600000 + 65536
    rng = np.random.default_rng(n + fm)
    # inputs of ranges far apart, so that a bound or a plan of the call before shows
    xs = [torch.from_numpy((10.0 ** k * rng.standard_normal(n)).astype(np.float32)).cuda() for k in (0, 3, -3)]

    def call(x, out, size, y, st):
        szp.compress_dev_async(x.data_ptr(), n, out.data_ptr(), cap, size.data_ptr(), szp.REL, 0.0, 1e-3, 32, T, fm, stream=st)
        szp.decompress_dev_async(out.data_ptr(), cap, size.data_ptr(), n, y.data_ptr(), 32, T, fm, stream=st)

    def body():
        want = []
        for x in xs:
            out = torch.zeros(cap, dtype=torch.uint8, device="cuda")
            y = torch.full((n,), float("nan"), device="cuda")
            torch.cuda.synchronize()
            sz = szp.compress_dev(x.data_ptr(), n, out.data_ptr(), cap, szp.REL, 0.0, 1e-3, 32, T, fm)
            szp.decompress_dev(out.data_ptr(), sz, n, y.data_ptr(), 32, T, fm)
            torch.cuda.synchronize()
            want.append((sz, out[:sz].clone(), y))
        s = torch.cuda.Stream()
        got = [(torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(cap, dtype=torch.uint8, device="cuda"),
                torch.full((n,), float("nan"), device="cuda")) for _ in xs]
        torch.cuda.synchronize()

        def all_calls():
            for x, (size, out, y) in zip(xs, got):
                call(x, out, size, y, s.cuda_stream)

        all_calls()
        s.synchronize()
        if graph:
            for size, out, y in got:
                size.zero_(), out.zero_(), y.fill_(float("nan"))
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s):
                all_calls()
            for _ in range(2):
                g.replay()
            torch.cuda.synchronize()
        for (sz, ref, ry), (size, out, y) in zip(want, got):
            assert int(size.item()) == sz
            assert torch.equal(out[:sz], ref)
            assert torch.equal(y.view(torch.int32), ry.view(torch.int32))

    _in_thread(body)  # a thread of its own: the library's buffers are a thread's
