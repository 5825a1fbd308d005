"""The ULV reduction by panels (``hss_factor_pan.cu``): every FP64 level, and FP32
levels with nodes of more than 128 rows.

Shapes at its edges: one and several panels of 32 reflectors (ranks 31 to 70), nodes
of 64 / 65, 128 / 129, 256 / 257 and 512 rows (register tiles, row tiles of 128,
chunks of 128 inner terms), ranks that differ between the sides, nodes with nothing
to eliminate, single leaves, and values over many decades.  FP64 solves against
the oracle to 1e-12; FP32 factors must refine to 1e-10 within three steps (a factor
good to FP32 gains six digits a step)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


SHAPES = [
    (130, 65, 31), (520, 130, 33), (258, 129, 64), (1030, 257, 70), (1024, 512, 40), (300, 150, 5), (500, 500, 8),
    (400, 13, 20),   # leaves of rank as large as their rows: nothing to eliminate
]


@pytest.mark.parametrize("n,ls,k", SHAPES)
def test_solves(pkg, orc, n, ls, k):
    rng = np.random.default_rng(n + k)
    h = orc.synthetic_hss(n, ls, k, rng)
    A = pkg.HssMatrix.from_tree(h)
    b = rng.standard_normal((n, 3))
    ref = orc.ulvfactsolve(h, b)
    F = pkg.ulvfactor(A, "fp64")
    assert rel(F.solve(b), ref) <= 1e-12
    F.refactor()
    assert rel(F.solve(b), ref) <= 1e-12
    st = {}
    z = pkg.ldiv(A, b, precision="fp32", tol=1e-10, stats=st)
    assert st["converged"] and st["iterations"] <= 3 and rel(z, ref) <= 1e-8


def test_uneven_ranks(pkg, orc):
    """Ranks of U and V drawn per node, as compression gives them."""
    n, ls = 700, 90
    rng = np.random.default_rng(3)
    cl = orc.bisection_cluster(n, ls)

    def orth(m, k):
        return np.linalg.qr(rng.standard_normal((m, k)))[0][:, :k]

    def build(t, root):
        if t.isleaf():
            m = len(t)
            ku, kv = rng.integers(5, 41, size=2)
            return orc.HssMatrix.leaf(rng.standard_normal((m, m)) / np.sqrt(m) + 4 * np.eye(m), orth(m, ku), orth(m, kv)), ku, kv
        a, ku1, kv1 = build(t.left, False)
        c, ku2, kv2 = build(t.right, False)
        B12, B21 = 0.1 * rng.standard_normal((ku1, kv2)), 0.1 * rng.standard_normal((ku2, kv1))
        if root:
            return orc.HssMatrix.branch(a, c, B12, B21, rootnode=True), 0, 0
        ku, kv = rng.integers(5, min(ku1 + ku2, 41)), rng.integers(5, min(kv1 + kv2, 41))
        R, W = orth(ku1 + ku2, ku), orth(kv1 + kv2, kv)
        return orc.HssMatrix.branch(a, c, B12, B21, R[:ku1], W[:kv1], R[ku1:], W[kv1:], rootnode=False), ku, kv

    h = build(cl, True)[0]
    A = pkg.HssMatrix.from_tree(h)
    b = rng.standard_normal((n, 2))
    assert rel(pkg.ldiv(A, b), orc.ulvfactsolve(h, b)) <= 1e-12


def test_scaled_rows_and_zero_blocks(pkg, orc):
    """Leaf rows scaled over 24 decades (products whose digits could do worse than an
    FP64 sum are summed in FP64) and zero rows of U (reflectors with tau = 0): the
    backward error, relative to each row's own size, stays at FP64's level."""
    n = 520
    rng = np.random.default_rng(6)
    h = orc.synthetic_hss(n, 130, 24, rng)

    def leaves(x):
        return [x] if x.leafnode else leaves(x.A11) + leaves(x.A22)

    scale = []
    for x in leaves(h):
        s = 10.0 ** rng.uniform(-12, 12, size=(x.D.shape[0], 1))
        x.D, x.U = s * x.D, s * x.U
        x.U[:30] = 0.0
        scale.append(s)
    s = np.vstack(scale)
    A = orc.full(h)
    b = s * rng.standard_normal((n, 2))
    x = pkg.ldiv(pkg.HssMatrix.from_tree(h), b)
    xo = orc.ulvfactsolve(h, b)

    def berr(v):
        return np.max(np.abs(A @ v - b) / (np.abs(A) @ np.abs(v) + np.abs(b)))

    assert berr(x) <= max(1e-12, 10 * berr(xo))


def test_singular_root_is_reported(pkg, orc):
    n = 300
    h = orc.synthetic_hss(n, 300, 8, np.random.default_rng(1))
    h.D[:, 7] = 0.0
    with pytest.raises(np.linalg.LinAlgError):
        pkg.matmul(pkg.HssMatrix.from_tree(h), np.ones(n))
        F = pkg.ulvfactor(pkg.HssMatrix.from_tree(h), "fp64")
        F.solve(np.ones(n))
