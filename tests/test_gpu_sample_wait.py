"""Waits of the tensor-core sample product that run out (HSS_OPT_POLL_LIMIT = 1): the
rows are NaN, the next call on the device reports HSS_ERR_TIMEOUT once, and products
after it are right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("r", [5, 40])
def test_runs_out(pkg, lib, r, trans):
    torch = pytest.importorskip("torch")
    L = pkg._lib
    m, n = 1500, 4100
    A = torch.randn((n, m) if trans else (m, n), dtype=torch.float64, device="cuda")
    D = pkg.DenseDevice(A)
    X = torch.randn(r, n, dtype=torch.float64, device="cuda")
    assert lib.hss_set_option(L.HSS_OPT_POLL_LIMIT, 1) == 0
    try:
        Y = pkg.sample(D, X, trans=trans)
        torch.cuda.synchronize()
    finally:
        lib.hss_set_option(L.HSS_OPT_POLL_LIMIT, 0)
    expired = bool(torch.isnan(Y).any())
    assert expired   # MMAs of a stage are not done at the first poll
    with pytest.raises(L.HssTimeout):
        pkg.sample(D, X, trans=trans)
    for _ in range(2):
        Y = pkg.sample(D, X, trans=trans)
        torch.cuda.synchronize()
        ref = ((A.T if trans else A) @ X.T).T
        assert float((Y - ref).norm() / ref.norm()) <= 1e-14
