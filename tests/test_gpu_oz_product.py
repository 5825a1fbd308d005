"""The tensor-core product (``hss_ozmv.cu``): taken by FP64 products of at least six
columns on matrices large enough, and by the refinement residual.

Shapes at the edges of its tiles: leaves of 127 to 130 and 300 rows (row tiles of
128, chunks of 128 inner terms), stacked translators of more than 128 rows and
inner terms, ranks that differ between the sides, column tiles of 16 and 32 with
remainders, single leaves, forests with an empty member.  Tolerances: 1e-12
against the oracle and 1e-13 against the level-by-level FP64 product, as for the
other products; entrywise K u |A| |x| (the bound of FP64 sums, K the terms of a
row's longest chain of sums) on data over many decades."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HSS_OPT_LEVEL_PRODUCT = 3
U = 2.0 ** -53


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def _level(lib, fn):
    assert lib.hss_set_option(HSS_OPT_LEVEL_PRODUCT, 1) == 0
    try:
        return fn()
    finally:
        lib.hss_set_option(HSS_OPT_LEVEL_PRODUCT, 0)


@pytest.mark.parametrize("n,ls,k,r", [
    (254, 127, 31, 500),     # two leaves of 127 rows, root only
    (520, 130, 17, 257),     # leaves of 130: two row tiles, two chunks; one column beyond a tile
    (600, 300, 70, 96),      # three row tiles, ranks above 64
    (1030, 65, 64, 130),     # stacked translators of 192 rows over 128 inner terms
    (200, 256, 8, 400),      # a single leaf
])
@pytest.mark.parametrize("trans", [False, True])
def test_edges(pkg, lib, orc, n, ls, k, r, trans):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + r)
    h = orc.synthetic_hss(n, ls, k, rng)
    dev = pkg.HssMatrix.from_tree(h).device()
    X = torch.from_numpy(rng.standard_normal((r, n))).cuda()
    C0 = torch.from_numpy(rng.standard_normal((r, n))).cuda()

    def run(alpha, beta):
        C = C0.clone()
        dev.matmul_device(X, n, r, C, n, alpha=alpha, beta=beta, trans=trans)
        torch.cuda.synchronize()
        return C.cpu().numpy().T

    A = orc.full(h)
    ref = (A.T if trans else A) @ X.cpu().numpy().T
    c0 = lib.hss_launch_counter()
    y = run(1.0, 0.0)
    assert n <= ls or lib.hss_launch_counter() - c0 > 1   # not one persistent launch
    assert rel(y, ref) <= 1e-12
    assert rel(y, _level(lib, lambda: run(1.0, 0.0))) <= 1e-13
    for alpha, beta in ((-1.0, 1.0), (0.5, -2.0), (2.0, 1.0)):
        z = run(alpha, beta)
        assert rel(z, alpha * ref + beta * C0.cpu().numpy().T) <= 1e-12


def test_forest_with_empty_member(pkg, lib, orc):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4)
    trees = [orc.synthetic_hss(n, ls, k, rng) for n, ls, k in
             [(1152, 64, 48), (640, 256, 20), (2001, 64, 16), (129, 64, 8), (64, 64, 8)]]
    dev = pkg.DeviceHss.from_trees([pkg.HssMatrix.from_tree(t) for t in trees])
    rs = [33, 7, 0, 16, 48]
    xs = [rng.standard_normal((r, t.size()[1])) for t, r in zip(trees, rs)]
    dX = [torch.from_numpy(x).cuda() for x in xs]
    dY = [torch.zeros_like(x) for x in dX]
    ns = [t.size()[0] for t in trees]
    dev.matmul_batch_device(dX, ns, rs, dY, ns)
    torch.cuda.synchronize()
    for t, x, y in zip(trees, xs, dY):
        if len(x):
            assert rel(y.cpu().numpy().T, orc.matmul(t, x.T)) <= 1e-12


def test_wide_range_and_not_finite(pkg, orc):
    """Entries over 40 decades (summed in FP64 where the digits would do worse), zero
    rows and columns; infinities and NaN reach the outputs they reach in FP64."""
    torch = pytest.importorskip("torch")
    n, r = 260, 300
    rng = np.random.default_rng(8)
    h = orc.synthetic_hss(n, 130, 12, rng)
    for leaf in (h.A11, h.A22):
        leaf.D *= 10.0 ** rng.uniform(-20, 20, size=leaf.D.shape)
        leaf.D[::7] = 0.0
    dev = pkg.HssMatrix.from_tree(h).device()
    X = rng.standard_normal((n, r)) * 10.0 ** rng.uniform(-10, 10, size=(n, r))
    X[:, 5] = 0.0
    ref, bound = [], []
    for f in (lambda a: a, np.abs):
        D1, D2, U1, U2, V1, V2, B12, B21 = (f(x).astype(np.longdouble) for x in (
            h.A11.D, h.A22.D, h.A11.U, h.A22.U, h.A11.V, h.A22.V, h.B12, h.B21))
        x1, x2 = f(X[:130]).astype(np.longdouble), f(X[130:]).astype(np.longdouble)
        ref.append(np.vstack([D1 @ x1 + U1 @ (B12 @ (V2.T @ x2)), D2 @ x2 + U2 @ (B21 @ (V1.T @ x1))]))
    bound = 400 * U * ref[1].astype(np.float64)

    def run(X):
        dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
        dY = torch.empty_like(dX)
        dev.matmul_device(dX, n, r, dY, n)
        torch.cuda.synchronize()
        return dY.cpu().numpy().T

    assert np.all(np.abs(run(X) - ref[0]) <= bound)
    X[3, 7], X[140, 9], X[200, 11] = np.inf, np.nan, -np.inf
    y = run(X)
    bad = np.zeros(r, dtype=bool)
    bad[[7, 9, 11]] = True
    assert np.all(np.isfinite(y[:, ~bad]))
    assert np.isnan(y[:, 9]).all()
    # 0 * inf in the zero rows of D, inf elsewhere in the leaf; NaN or inf through the coupling
    assert not np.isfinite(y[:, 7]).any() and not np.isfinite(y[:, 11]).any()
