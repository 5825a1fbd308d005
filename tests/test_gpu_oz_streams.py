"""The tensor-core product's digit slices, made once per plan on the stream of the call that
needs them first (of these products the second on a plan): calls on other streams and threads wait for them, and a stream that the caller captures
makes none.  Against the oracle: products 1e-12, solves 1e-10 by the residual."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, LS, K, R = 16384, 128, 32, 32
MV_DX = 8


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.fixture(scope="module")
def tree(orc):
    return orc.synthetic_hss(N, LS, K, np.random.default_rng(5))


def _columns(torch, b, stream):
    with torch.cuda.stream(stream):
        d = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
        out = d, torch.zeros_like(d)
    stream.synchronize()
    return out


def test_other_stream(pkg, orc, tree):
    """The stream of the product that makes them is busy when a solve on another one needs the slices."""
    torch = pytest.importorskip("torch")
    dev = pkg.DeviceHss(pkg.HssMatrix.from_tree(tree))
    b = np.random.default_rng(1).standard_normal((N, R))
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    x, y = _columns(torch, b, one)
    rhs, sol = _columns(torch, b, two)
    F = dev.ulvfactor("fp32", stream=two)
    two.synchronize()
    dev.matmul_device(x, N, R, y, N, stream=one)
    with torch.cuda.stream(one):
        torch.cuda._sleep(100_000_000)   # about 50 ms
    dev.matmul_device(x, N, R, y, N, stream=one)
    F.solve_device(rhs, N, R, sol, N, tol=1e-10, stream=two)
    two.synchronize()
    res = np.linalg.norm(b - orc.matmul(tree, sol.cpu().numpy().T), axis=0) / np.linalg.norm(b, axis=0)
    assert res.max() <= 1e-10
    one.synchronize()
    assert rel(y.cpu().numpy().T, orc.matmul(tree, b)) <= 1e-12


def test_other_threads(pkg, orc, tree):
    """Two factorizations of one plan, each solved with on its own thread and stream."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(2)
    for _turn in range(3):
        dev = pkg.DeviceHss(pkg.HssMatrix.from_tree(tree))
        jobs = []
        for _ in range(2):
            st, b = torch.cuda.Stream(), rng.standard_normal((N, 4))
            jobs.append((st, b, dev.ulvfactor("fp32", stream=st)) + _columns(torch, b, st))
        errors = []

        def work(job):
            try:
                st, _b, F, rhs, sol = job
                F.solve_device(rhs, N, 4, sol, N, tol=1e-10, stream=st)
                st.synchronize()
            except Exception as e:   # noqa: BLE001
                errors.append(e)

        threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors
        for _st, b, _F, _rhs, sol in jobs:
            res = np.linalg.norm(b - orc.matmul(tree, sol.cpu().numpy().T)) / np.linalg.norm(b)
            assert res <= 1e-10


def test_capture(pkg, lib, orc, tree):
    """A captured product after others on the same plan: with the slices it replays
    the tensor-core product; where their buffer could not be had, the capture makes no
    allocation and holds the other product."""
    torch = pytest.importorskip("torch")
    L = pkg._lib
    b = np.random.default_rng(3).standard_normal((N, R))
    ref = orc.matmul(tree, b)
    for slices in (True, False):
        dev = pkg.DeviceHss(pkg.HssMatrix.from_tree(tree))
        st = torch.cuda.Stream()
        x, y = _columns(torch, b, st)
        dev.matmul_device(x, N, R, y, N, stream=st)
        if not slices:
            assert lib.hss_set_option(L.HSS_OPT_FAIL_ALLOC, 1) == 0
        try:
            pkg.linalg.trace_begin(MV_DX)
            dev.matmul_device(x, N, R, y, N, stream=st)
            st.synchronize()
            assert (pkg.linalg.trace_end()[1] > 0) == slices
        finally:
            lib.hss_set_option(L.HSS_OPT_FAIL_ALLOC, 0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            dev.matmul_device(x, N, R, y, N, stream=st)
        y.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert rel(y.cpu().numpy().T, ref) <= 1e-12
