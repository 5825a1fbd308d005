"""Factorizations whose pivots have no finite reciprocal: a single block of small integers
scaled to the subnormal range of its precision (and one near the largest numbers, whose
reciprocals are).  The elimination and both substitutions then divide.  Entries keep 44 bits in FP64 and 14 in FP32; solutions within 1e-10 and
1e-1 of the one that the right-hand side was made from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 40, 100, 200])
@pytest.mark.parametrize("prec,scale,tol", [("fp64", -1030, 1e-10), ("fp32", -135, 1e-1), ("fp64", 1000, 1e-12)])
def test_scaled_block(pkg, orc, n, prec, scale, tol):
    rng = np.random.default_rng(n)
    # diagonally dominant (no growth), small integers: exact in either range
    M = rng.integers(-1, 2, (n, n)).astype(float)
    M[np.arange(n), np.arange(n)] = 0.0
    keep = rng.random((n, n)) < 4.0 / n
    M = M * keep + np.diag(rng.permutation(np.arange(n)) % 8 + 12.0)
    x = rng.integers(-3, 4, (n, 3)).astype(float)
    D, b = np.ldexp(M, scale), np.ldexp(M @ x, scale)
    F = pkg.HssMatrix.from_tree(orc.HssMatrix.leaf(D, rootnode=True)).device().ulvfactor(prec)
    got = F.solve(b, tol=-1.0)
    assert np.abs(got - x).max() <= tol


@pytest.mark.parametrize("prec,scale,tol", [("fp64", -1015, 1e-10), ("fp32", -115, 1e-3)])
@pytest.mark.parametrize("n,ls,k,r", [(700, 64, 8, 4), (4096, 64, 16, 40), (1500, 250, 20, 3)])
def test_tiny_and_infinite_columns(pkg, orc, n, ls, k, r, prec, scale, tol):
    """Right-hand sides next to each other: ordinary, so small that a quotient's correction
    underflows, and with an infinite and a NaN entry.  The first two are solved as ever
    (their scaled solutions to the tolerance of an unrefined solve), the others give
    no finite solution."""
    rng = np.random.default_rng(n)
    h = orc.synthetic_hss(n, ls, k, rng)
    b = rng.standard_normal((n, r))
    ref = orc.ulvfactsolve(h, b)
    tiny = np.arange(r) % 2 == 1
    b[:, tiny] = np.ldexp(b[:, tiny], scale)
    b[n // 3, r - 1] = np.inf
    b[n // 2, r - 2] = np.nan
    x = pkg.HssMatrix.from_tree(h).device().ulvfactor(prec).solve(b, tol=-1.0)
    assert not np.isfinite(x[:, r - 2:]).any(axis=0).all()
    x[:, tiny] = np.ldexp(x[:, tiny], -scale)
    for j in range(r - 2):
        assert np.linalg.norm(x[:, j] - ref[:, j]) <= tol * np.linalg.norm(ref[:, j]), j
