"""Rounding of the flat product: a row of D x is added up in runs of 16 terms (of 8 where
there are at most 64), not in one chain.  With normal entries a sum of j terms has
variance j and an addition to it an error of 0.425 units of roundoff u of it (rms).  So
128 terms in one chain have an rms error of 3.4 u relative to their sum's rms, in eight
runs of 16 added one by one 1.5 u; 64 terms 2.4 u, in eight runs of 8 1.1 u; with the
last rounding below 1.7 and 1.3 u.  The lines are between them; 8192 rows and every
count of columns give the rms to 1 %."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("ls,bound", [(128, 2.4), (64, 1.8)])
@pytest.mark.parametrize("r", [1, 2, 3, 4])
def test_rows_in_runs(pkg, orc, ls, bound, r):
    torch = pytest.importorskip("torch")
    n = 8192
    rng = np.random.default_rng(r)
    h = orc.synthetic_hss(n, ls, 8, rng)
    leaves, stack = [], [h]
    while stack:
        x = stack.pop()
        if x.leafnode:
            leaves.append(x)
        else:
            stack += [x.A22, x.A11]
    X = rng.standard_normal((n, r))
    ref, row = np.empty((n, r), dtype=np.longdouble), 0
    for x in leaves:   # D alone: U = 0
        x.U[:] = 0.0
        x.D[:] = rng.standard_normal(x.D.shape)
        m = x.D.shape[0]
        ref[row:row + m] = x.D.astype(np.longdouble) @ X[row:row + m].astype(np.longdouble)
        row += m
    assert row == n
    dev = pkg.HssMatrix.from_tree(h).device()
    dX = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
    dY = torch.empty_like(dX)
    dev.matmul_device(dX, n, r, dY, n)
    err = dY.cpu().numpy().T.astype(np.longdouble) - ref
    rms = float(np.sqrt(np.sum(err ** 2) / np.sum(ref ** 2)))
    assert rms < bound * U, rms / U
