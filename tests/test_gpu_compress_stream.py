"""Adaptive compression called while the caller's current stream is not the default
one: the sample products (on the default stream) and the tensor operations between
them (on the caller's) are ordered, so that the result is the default stream's, bit
for bit (the same kernels on the same draws)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_adaptive_on_another_stream(pkg, orc):
    import torch
    from hssmatrices_gb300 import compression as CP

    n = 8192
    A = CP.DenseDevice(orc.cauchy_matrix(n))
    cl = pkg.bisection_cluster(n, 128)
    x = np.random.default_rng(2).standard_normal((n, 2))

    def run():
        st = {}
        dev = pkg.randcompress_adaptive(A, cl, cl, kest=10, atol=1e-9, rtol=1e-9, noversampling=10, stepsize=20,
                                        rng=np.random.default_rng(1), device=True, stats=st)
        return st["rounds"], st["ranks"], dev.matmul_host(x)

    ref = run()
    torch.cuda.synchronize()
    assert ref[0] >= 2   # a round that failed: its row test columns join the sample
    side = torch.cuda.Stream()
    for _ in range(3):
        with torch.cuda.stream(side):
            out = run()
        torch.cuda.synchronize()
        assert out[0] == ref[0] and np.array_equal(out[1], ref[1]) and np.array_equal(out[2], ref[2])
