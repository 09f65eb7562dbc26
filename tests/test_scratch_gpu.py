"""GPU: scratch from the library's pool, shared by streams and threads, given back on request."""
import threading

import numpy as np
import pytest
import torch

import morpheus_gb300 as mgb
from morpheus_gb300 import _lib
from morpheus_gb300 import generators as gen

pytestmark = pytest.mark.gpu


def test_threads_and_streams_share_the_pool(cuda):
    A = mgb.matrix_from_host(gen.csr_to_coo_host(gen.power_law(30_000, seed=3)))
    xs = [torch.rand(30_000, dtype=torch.float64, device="cuda") for _ in range(4)]
    want = []
    for x in xs:
        y = torch.empty_like(x)
        mgb.multiply(A, x, y)
        want.append((y, mgb.dot(30_000, x, y)))
    torch.cuda.synchronize()
    failed = []

    def work(k):
        s = torch.cuda.Stream()
        y = torch.empty_like(xs[k])
        s.wait_stream(torch.cuda.current_stream())
        for _ in range(50):
            mgb.multiply(A, xs[k], y, stream=s)
            if mgb.dot(30_000, xs[k], y, stream=s) != want[k][1] or not torch.equal(y, want[k][0]):
                failed.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_release_and_use_again(cuda):
    x = torch.rand(100_000, dtype=torch.float64, device="cuda")
    a = mgb.dot(100_000, x, x)
    _lib.call("mgb_scratch_release")
    _lib.call("mgb_scratch_release")
    assert mgb.dot(100_000, x, x) == a
    assert abs(a - float((x.cpu().numpy() ** 2).sum())) <= 1e-12 * a


def test_scratch_under_capture(cuda):
    hm = gen.csr_to_coo_host(gen.power_law(5000, seed=4))
    A = mgb.matrix_from_host(hm)
    x = torch.rand(5000, dtype=torch.float64, device="cuda")
    y, want = torch.empty_like(x), torch.empty_like(x)
    mgb.multiply(A, x, want)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        mgb.multiply(A, x, y, stream=s)
    for _ in range(3):
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), want.cpu().numpy())
