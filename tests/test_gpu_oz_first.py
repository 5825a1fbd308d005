"""Which product the first ones on a plan take (``oz_first_pays``): slices are made at once
where they pay within that product or are small, else from the second product on; slices
that a refined solve has made are used at once.  All of them against the oracle, 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MV_DX = 8


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.fixture(scope="module")
def large(orc):
    return orc.synthetic_hss(65536, 128, 32, np.random.default_rng(9))


@pytest.fixture(scope="module")
def small(orc):
    return orc.synthetic_hss(520, 130, 17, np.random.default_rng(9))


@pytest.mark.parametrize("size,r,taken", [
    ("large", 6, [False, True, True]),
    ("large", 32, [True, True]),
    ("large", 4, [False, False, False]),    # the flat product every time
    ("small", 257, [True, True]),
])
def test_taken(pkg, orc, request, size, r, taken):
    torch = pytest.importorskip("torch")
    h = request.getfixturevalue(size)
    n = h.size()[0]
    dev = pkg.DeviceHss(pkg.HssMatrix.from_tree(h))
    x = np.random.default_rng(r).standard_normal((n, r))
    ref = orc.matmul(h, x)
    X = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    Y = torch.empty_like(X)
    for want in taken:
        pkg.linalg.trace_begin(MV_DX)
        dev.matmul_device(X, n, r, Y, n)
        torch.cuda.synchronize()
        assert (pkg.linalg.trace_end()[1] > 0) == want
        assert rel(Y.cpu().numpy().T, ref) <= 1e-12


def test_slices_of_a_solve(pkg, orc, large):
    torch = pytest.importorskip("torch")
    n = large.size()[0]
    dev = pkg.DeviceHss(pkg.HssMatrix.from_tree(large))
    x = np.random.default_rng(2).standard_normal((n, 6))
    dev.ulvfactor("fp32").solve(x, tol=1e-10)
    X = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    Y = torch.empty_like(X)
    pkg.linalg.trace_begin(MV_DX)
    dev.matmul_device(X, n, 6, Y, n)
    torch.cuda.synchronize()
    assert pkg.linalg.trace_end()[1] > 0
    assert rel(Y.cpu().numpy().T, orc.matmul(large, x)) <= 1e-12
