"""The tensor-core product on trees with levels of rank 0 (``hss_ozmv.cu``).

Such a level's launch has no work, and the launches are programmatic dependents of
each other: a grid without units still has to wait for the one before it, or the
launch after it reads the workspace and C too early.  512 leaves, so that the leaf
launch fills the SMs, each product several times on other columns; products against
the oracle (1e-12, as for the others), solves by the oracle's residual (twice the
tolerance that the solve was asked for)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MV_DX = 8
N, LS = 65536, 128


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def _orth(rng, m, k):
    return np.linalg.qr(rng.standard_normal((m, max(min(k, m), 0))))[0] if min(m, k) else np.zeros((m, k))


def ranked(orc, rng, rank):
    """A tree whose nodes of depth d have rank(d) (0 x k translators below a rank of 0)."""
    def build(cl, d):
        k = 0 if d == 0 else rank(d)
        if cl.isleaf():
            m = len(cl)
            D = rng.standard_normal((m, m)) / np.sqrt(m) + 4.0 * np.eye(m)
            return orc.HssMatrix.leaf(D, _orth(rng, m, k), _orth(rng, m, k), rootnode=False), k
        a, ka = build(cl.left, d + 1)
        b, kb = build(cl.right, d + 1)
        B12, B21 = (0.5 * rng.standard_normal(s) / np.sqrt(max(ka, 1)) for s in ((ka, kb), (kb, ka)))
        if d == 0:
            return orc.HssMatrix.branch(a, b, B12, B21, rootnode=True), 0
        R, W = (_orth(rng, ka + kb, k) for _ in range(2))
        return orc.HssMatrix.branch(a, b, B12, B21, R[:ka], W[:ka], R[ka:], W[ka:], rootnode=False), k
    return build(orc.bisection_cluster(N, LS), 0)[0]


RANKS = {
    "all": lambda d: 0,
    "root": lambda d: 0 if d <= 1 else 16,            # two matrices side by side
    "upper": lambda d: 0 if d <= 4 else 16,           # several empty levels in a row
    "middle": lambda d: 0 if d == 4 else 16,          # rank 0 between ranks of 16 (a product only)
}


@pytest.fixture(scope="module", params=sorted(RANKS))
def tree(request, pkg, orc):
    h = ranked(orc, np.random.default_rng(len(request.param)), RANKS[request.param])
    return request.param, h, pkg.HssMatrix.from_tree(h).device()


@pytest.mark.parametrize("r", [6, 32])
def test_product(pkg, orc, tree, r):
    torch = pytest.importorskip("torch")
    _name, h, dev = tree
    rng = np.random.default_rng(r)
    X = [rng.standard_normal((N, r)) for _ in range(4)]
    dX = [torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in X]
    C0 = torch.from_numpy(rng.standard_normal((r, N))).cuda()
    out = []
    pkg.linalg.trace_begin(MV_DX)
    for _ in range(3):
        for x in dX:
            C = C0.clone()
            dev.matmul_device(x, N, r, C, N, alpha=-1.0, beta=0.5)
            out.append(C)
    torch.cuda.synchronize()
    assert pkg.linalg.trace_end()[1] > 0   # the tensor-core product ran
    for i, x in enumerate(X):
        ref = 0.5 * C0.cpu().numpy().T - orc.matmul(h, x)
        for C in out[i::4]:
            assert rel(C.cpu().numpy().T, ref) <= 1e-12


def test_refined_solve(pkg, orc, tree):
    name, h, dev = tree
    if name == "middle":
        pytest.skip("a node without rows has no ULV reduction of rank 16")
    F = dev.ulvfactor("fp32")
    rng = np.random.default_rng(3)
    for r in (3, 32):
        b = rng.standard_normal((N, r))
        x = F.solve(b, tol=1e-12, maxit=20)
        res = np.linalg.norm(b - orc.matmul(h, x), axis=0) / np.linalg.norm(b, axis=0)
        assert res.max() <= 2e-12
