"""The groups of the flat product (``hss_flat.cu``): trees with fewer and more leaves
than SMs (groups of 1, 2, 4 and 8 leaves), a second pass over the groups, uneven trees,
ranks of 64 (two staged translators instead of three), chunks of one to four columns,
up to 32 columns, the adjoint, alpha and beta.

Against the oracle and the queued product: sums of at most 2^15 products of entries
of order one, relative (2-norm) 1e-12 and 1e-13 as for the other product paths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HSS_OPT_FLAT_PRODUCT = 6


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("n,ls,k,rs", [
    (90, 45, 7, (1, 3, 32)),             # two leaves: no branch above the groups
    (700, 50, 20, (1, 5, 6, 7, 32)),     # groups of one, chunks of one column
    (2600, 13, 6, (1, 2, 4, 9)),         # 256 leaves
    (5000, 9, 4, (1, 4)),                # 1024 leaves: groups of eight
    (20480, 20, 16, (2, 5)),             # ... and two passes over them
    (4096, 64, 64, (1, 4, 8)),           # ranks of 64
    (1030, 257, 40, (1, 11)),            # leaves of more than 256 rows
])
def test_groups(pkg, lib, orc, n, ls, k, rs):
    rng = np.random.default_rng(n)
    h = orc.synthetic_hss(n, ls, k, rng)
    A = pkg.HssMatrix.from_tree(h)
    for r in rs:
        x = rng.standard_normal((n, r))
        y = pkg.matmul(A, x)
        assert rel(y, orc.matmul(h, x)) <= 1e-12
        assert np.array_equal(pkg.matmul(A, x), y)
        C0 = np.asfortranarray(rng.standard_normal((n, r)))
        C = C0.copy(order="F")
        pkg.mul(C, A, x, -1.5, 0.25)
        assert rel(C, orc.matmul(h, x, -1.5, 0.25, C0)) <= 1e-12
        lib.hss_set_option(HSS_OPT_FLAT_PRODUCT, 0)
        try:
            assert rel(y, pkg.matmul(A, x)) <= 1e-13
        finally:
            lib.hss_set_option(HSS_OPT_FLAT_PRODUCT, 1)


@pytest.mark.parametrize("r", [1, 6])
def test_groups_of_a_comb(pkg, orc, r):
    """A tree that is deep on one side: groups of different sizes and heights."""
    rng = np.random.default_rng(4)
    sizes = [40, 33, 65, 20, 48, 64, 31, 50, 27, 36, 44, 52, 61]
    k = 12

    def orth(m):
        return np.linalg.qr(rng.standard_normal((m, k)))[0]

    def leaf(m):
        return orc.HssMatrix.leaf(rng.standard_normal((m, m)) + 4 * np.eye(m), orth(m), orth(m))

    h = leaf(sizes[0])
    for i, m in enumerate(sizes[1:]):
        b = [0.1 * rng.standard_normal((k, k)) for _ in range(2)]
        if i == len(sizes) - 2:
            h = orc.HssMatrix.branch(h, leaf(m), *b, rootnode=True)
        else:
            R, W = orth(2 * k), orth(2 * k)
            h = orc.HssMatrix.branch(h, leaf(m), *b, R[:k], W[:k], R[k:], W[k:])
    x = rng.standard_normal((sum(sizes), r))
    assert rel(pkg.matmul(pkg.HssMatrix.from_tree(h), x), orc.matmul(h, x)) <= 1e-12
