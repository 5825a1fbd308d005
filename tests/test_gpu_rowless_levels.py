"""Levels whose nodes have no rows left but carry column bases: children of row rank 0
and column rank above 0, and the other way round.  A level of such nodes alone sizes the
one-block factor kernel's shared memory.  Solutions against the oracle (1e-12 for FP64,
1e-8 refined)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _orth(rng, m, k):
    return np.linalg.qr(rng.standard_normal((m, k)))[0] if m and k else np.zeros((m, k))


def build(orc, rng, rows, depth, ku, kv):
    """A chain of branches on the left, `depth` of them below the root; ku(height), kv(height)."""
    def leaf(h):
        D = rng.standard_normal((rows, rows)) / np.sqrt(rows) + 4.0 * np.eye(rows)
        return orc.HssMatrix.leaf(D, _orth(rng, rows, ku(h)), _orth(rng, rows, kv(h)), rootnode=False)

    node, u, v = leaf(0), ku(0), kv(0)
    for h in range(1, depth + 2):
        other = leaf(0)
        B12 = 0.3 * rng.standard_normal((u, kv(0)))
        B21 = 0.3 * rng.standard_normal((ku(0), v))
        if h == depth + 1:
            return orc.HssMatrix.branch(node, other, B12, B21, rootnode=True)
        un, vn = min(ku(h), u + ku(0)), min(kv(h), v + kv(0))
        R, W = _orth(rng, u + ku(0), un), _orth(rng, v + kv(0), vn)
        node = orc.HssMatrix.branch(node, other, B12, B21, R[:u], W[:v], R[u:], W[v:], rootnode=False)
        u, v = un, vn


@pytest.mark.parametrize("rows", [20, 60, 150])
@pytest.mark.parametrize("ku,kv", [
    (lambda h: 0, lambda h: 5),
    (lambda h: 0, lambda h: 18),
    (lambda h: 6, lambda h: 0),
    (lambda h: 7 if h == 0 else 0, lambda h: 4),
])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-8)])
def test_factor_and_solve(pkg, lib, orc, rows, ku, kv, prec, tol):
    rng = np.random.default_rng(rows)
    h = build(orc, rng, rows, 4, ku, kv)
    n = h.size()[0]
    b = rng.standard_normal((n, 3))
    ref = orc.ulvfactsolve(h, b)
    F = pkg.HssMatrix.from_tree(h).device().ulvfactor(prec)
    x = F.solve(b, tol=1e-11 if prec == "fp32" else 0.0)
    assert np.linalg.norm(x - ref) <= tol * np.linalg.norm(ref)
