"""Values at the ends of the range in the tensor-core product (``hss_ozmv.cu``), at sizes
that take it (asserted by its leaf launch): entries over 40 decades, which the digits do
worse than FP64 and the kernel sums in FP64, zero rows and columns, infinities and NaN;
and a single leaf, whose product is the leaf launch alone.  Entrywise K u |A| |x| with K
the terms of a row's chain of sums, below 400."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MV_DX = 8
U = 2.0 ** -53


def product(pkg, torch, dev, X, n, **kw):
    dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    dY = torch.empty_like(dX)
    pkg.linalg.trace_begin(MV_DX)
    dev.matmul_device(dX, n, X.shape[1], dY, n, **kw)
    torch.cuda.synchronize()
    assert pkg.linalg.trace_end()[1] == 1
    return dY.cpu().numpy().T


@pytest.mark.parametrize("r", [400, 449])
def test_wide_range_and_not_finite(pkg, orc, r):
    torch = pytest.importorskip("torch")
    n = 260
    rng = np.random.default_rng(r)
    h = orc.synthetic_hss(n, 130, 16, rng)
    for leaf in (h.A11, h.A22):
        leaf.D *= 10.0 ** rng.uniform(-20, 20, size=leaf.D.shape)
        leaf.D[::7] = 0.0
    dev = pkg.HssMatrix.from_tree(h).device()
    X = rng.standard_normal((n, r)) * 10.0 ** rng.uniform(-10, 10, size=(n, r))
    X[:, 5] = 0.0
    ref = []
    for f in (lambda a: a, np.abs):
        D1, D2, U1, U2, V1, V2, B12, B21 = (f(x).astype(np.longdouble) for x in (
            h.A11.D, h.A22.D, h.A11.U, h.A22.U, h.A11.V, h.A22.V, h.B12, h.B21))
        x1, x2 = f(X[:130]).astype(np.longdouble), f(X[130:]).astype(np.longdouble)
        ref.append(np.vstack([D1 @ x1 + U1 @ (B12 @ (V2.T @ x2)), D2 @ x2 + U2 @ (B21 @ (V1.T @ x1))]))
    bound = 400 * U * ref[1].astype(np.float64)
    assert np.all(np.abs(product(pkg, torch, dev, X, n) - ref[0]) <= bound)
    X[3, 7], X[140, 9], X[200, 11] = np.inf, np.nan, -np.inf
    y = product(pkg, torch, dev, X, n)
    good = np.ones(r, dtype=bool)
    good[[7, 9, 11]] = False
    assert np.all(np.abs(y - ref[0])[:, good] <= bound[:, good])
    assert np.isnan(y[:, 9]).all()
    # 0 * inf in the zero rows of D, inf elsewhere in the leaf; NaN or inf through the coupling
    assert not np.isfinite(y[:, [7, 11]]).any()


@pytest.mark.parametrize("scale", [0, 300, -300])
def test_scaled(pkg, orc, scale):
    """Couplings and vectors at the ends of FP64's range: scaling by powers of two is exact."""
    torch = pytest.importorskip("torch")
    n, r = 260, 400
    rng = np.random.default_rng(3)
    h = orc.synthetic_hss(n, 130, 16, rng)
    X = rng.standard_normal((n, r))
    ref = orc.matmul(h, X)
    for leaf in (h.A11, h.A22):
        leaf.D = np.ldexp(leaf.D, 2 * scale)
    h.B12, h.B21 = np.ldexp(h.B12, 2 * scale), np.ldexp(h.B21, 2 * scale)
    dev = pkg.HssMatrix.from_tree(h).device()
    y = np.ldexp(product(pkg, torch, dev, np.ldexp(X, scale), n), -3 * scale)
    assert np.linalg.norm(y - ref) <= 1e-14 * np.linalg.norm(ref)


@pytest.mark.parametrize("trans", [False, True])
def test_single_leaf(pkg, orc, trans):
    torch = pytest.importorskip("torch")
    n, r = 200, 1200
    rng = np.random.default_rng(4)
    D = rng.standard_normal((n, n)) * 10.0 ** rng.uniform(-15, 15, size=(n, n))
    D[:, 3] = 0.0
    dev = pkg.HssMatrix.from_tree(orc.HssMatrix.leaf(D, rootnode=True)).device()
    X = rng.standard_normal((n, r))
    A = D.T if trans else D
    y = product(pkg, torch, dev, X, n, trans=trans)
    ref = A.astype(np.longdouble) @ X.astype(np.longdouble)
    assert np.all(np.abs(y - ref) <= n * U * (np.abs(A) @ np.abs(X)))
