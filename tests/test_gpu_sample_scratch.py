"""The sample product where the tensor-core kernel's scratch cannot be allocated
(HSS_OPT_FAIL_ALLOC): the CUDA cores' product takes the call, as it did before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-0.5, 2.0)])
def test_without_scratch(pkg, lib, trans, alpha, beta):
    torch = pytest.importorskip("torch")
    L = pkg._lib
    m, n, r = 900, 3000, 11
    A = torch.randn((n, m) if trans else (m, n), dtype=torch.float64, device="cuda")
    D = pkg.DenseDevice(A)
    X = torch.randn(r, n, dtype=torch.float64, device="cuda")
    Y0 = torch.randn(r, m, dtype=torch.float64, device="cuda")
    ref = alpha * ((A.T if trans else A) @ X.T).T + beta * Y0
    c0 = lib.hss_launch_counter()
    for fail, launches in ((0, (2, 3)), (1, (1, 2))):   # slices, product, sums; product, sums
        assert lib.hss_set_option(L.HSS_OPT_FAIL_ALLOC, fail) == 0
        try:
            Y = pkg.sample(D, X, trans=trans, out=Y0.clone(), alpha=alpha, beta=beta)
        finally:
            lib.hss_set_option(L.HSS_OPT_FAIL_ALLOC, 0)
        c1 = lib.hss_launch_counter()
        assert c1 - c0 in launches
        c0 = c1
        assert float((Y - ref).norm() / ref.norm()) <= 1e-14
