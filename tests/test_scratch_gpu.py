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


# around the one-launch limit (131,072), fewer elements than threads or vectors, and views that 16-byte loads cannot take
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1, 3, 8, 4095, 16387, 131071, 131072, 131073])
def test_short_reductions(cuda, n, dtype):
    import math
    rng = np.random.default_rng(n)
    x, y = (rng.uniform(-1, 1, n + 1).astype(dtype) for _ in range(2))
    xt, yt = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    # a thread adds at most 16 elements of each of 4 sums, then 2 + 5 + 4 + 7 levels: 64 roundings at most
    tol = 64 * np.finfo(dtype).eps
    for a, b in ((0, n), (1, n + 1)):
        u, v = x[a:b].astype(np.float64), y[a:b].astype(np.float64)
        ut, vt = xt[a:b], yt[a:b]
        size = math.fsum(np.abs(u * v))
        assert abs(mgb.dot(n, ut, vt) - math.fsum(u * v)) <= tol * size
        assert abs(mgb.dot(n, ut, ut) - math.fsum(u * u)) <= tol * math.fsum(u * u)
        assert abs(mgb.reduce(ut, n) - math.fsum(u)) <= tol * math.fsum(np.abs(u))
        assert mgb.dot(n, ut, vt) == mgb.dot(n, ut, vt)


@pytest.mark.parametrize("n", [1, 31, 700])
def test_short_reductions_beside_other_work(cuda, n):
    """CTAs of the cluster that have nothing to add, started while other kernels hold most of the GPU."""
    x = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
    big, side = torch.ones(1 << 24, device="cuda"), torch.cuda.Stream()
    out = torch.empty(200, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for k in range(200):
        big.mul_(1.0)
        with torch.cuda.stream(side):
            _lib.call("mgb_reduce_f64_async", x.data_ptr(), n, out[k:].data_ptr(), side.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(out, torch.full_like(out, n * (n + 1) / 2))
