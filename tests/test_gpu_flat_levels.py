"""The flat product over all its column counts: a plan holds the groups of the sizes that
some count takes, so every count from 1 to 32 has to find its own (trees of 8, 64
and 512 leaves, which take single leaves, groups of 1 to 4, and of 4 and 8).  Against the oracle, 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ls,k", [(512, 64, 16), (3000, 64, 20), (20011, 40, 12)])
@pytest.mark.parametrize("trans", [False, True])
def test_every_count(pkg, lib, orc, n, ls, k, trans):
    torch = pytest.importorskip("torch")
    h = orc.synthetic_hss(n, ls, k, np.random.default_rng(n))
    dev = pkg.HssMatrix.from_tree(h).device()
    x = np.random.default_rng(1).standard_normal((n, 32))
    ref = orc.matmul(orc.adjoint(h) if trans else h, x)
    X = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    for r in range(1, 33):
        Y = torch.zeros((r, n), dtype=torch.float64, device="cuda")
        dev.matmul_device(X, n, r, Y, n, trans=trans)
        y = Y.cpu().numpy().T
        assert np.linalg.norm(y - ref[:, :r]) <= 1e-12 * np.linalg.norm(ref[:, :r]), r
