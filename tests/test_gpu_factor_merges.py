"""The reduction of FP32 levels of at most 64 x 64 nodes and FP64 levels of at most
40 x 40 (``hss_factor_blk.cu``), one mbarrier per reflector, and solve lists that hold
nodes on both sides of 64 rows.

Ranks at the edges of the 32-reflector panel and of the 8-lane groups (a rank of 33
takes the general path), nodes of 62 to 66 rows, and forests of trees of different
heights, whose downward lists hold 128-row leaves beside 64 x 64 branches.  An FP32
factor is good to six digits of these well-conditioned matrices, so one solve without
refinement has to be within 1e-4 of the oracle's, and refinement reaches 1e-10
within three steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("n,ls,k", [(1024, 128, 32), (1024, 128, 33), (1024, 128, 31), (512, 64, 16), (600, 50, 7),
                                    (520, 65, 32), (260, 32, 1)])
def test_merges(pkg, orc, n, ls, k):
    rng = np.random.default_rng(n + k)
    h = orc.synthetic_hss(n, ls, k, rng)
    b = rng.standard_normal((n, 5))
    ref = orc.ulvfactsolve(h, b)
    F = pkg.ulvfactor(pkg.HssMatrix.from_tree(h), "fp32")
    for _ in range(2):
        assert rel(F.solve(b, tol=1e-10, maxit=3), ref) <= 1e-8   # raises unless it converged
        F.refactor()


@pytest.mark.parametrize("n,ls,k", [(512, 64, 16), (600, 50, 7), (260, 32, 1), (320, 20, 16), (512, 64, 17),
                                    (320, 40, 8), (320, 40, 7), (328, 41, 9), (320, 40, 33)])
def test_merges_fp64(pkg, orc, n, ls, k):
    """FP64 levels of at most 40 x 40 nodes (ranks of 7 and 33 at 40 rows have more than
    one panel and go to the panel kernels, as do 41 rows): 1e-12."""
    rng = np.random.default_rng(n + k)
    h = orc.synthetic_hss(n, ls, k, rng)
    b = rng.standard_normal((n, 3))
    ref = orc.ulvfactsolve(h, b)
    F = pkg.ulvfactor(pkg.HssMatrix.from_tree(h), "fp64")
    for _ in range(2):
        assert rel(F.solve(b), ref) <= 1e-12
        F.refactor()


@pytest.mark.parametrize("shapes", [[(2048, 128, 32), (1024, 128, 16)], [(700, 90, 20), (300, 40, 9), (128, 128, 8)]])
def test_heights(pkg, orc, shapes):
    import torch

    rng = np.random.default_rng(11)
    hs = [orc.synthetic_hss(n, ls, k, rng) for n, ls, k in shapes]
    bs = [rng.standard_normal((n, 4)) for n, _, _ in shapes]
    refs = [orc.ulvfactsolve(h, b) for h, b in zip(hs, bs)]
    F = pkg.DeviceHss.from_trees([pkg.HssMatrix.from_tree(h) for h in hs]).ulvfactor("fp32")
    dB = [torch.from_numpy(np.ascontiguousarray(b.T)).cuda() for b in bs]
    dX = [torch.empty_like(x) for x in dB]
    ns = [b.shape[0] for b in bs]
    F.solve_batch_device(dB, ns, [4] * len(ns), dX, ns, tol=-1.0)
    torch.cuda.synchronize()
    for x, ref in zip(dX, refs):
        assert rel(x.cpu().numpy().T, ref) <= 1e-4
