"""Batches of matrices whose levels hold several size classes, in every order of the
matrices: leaves of 128, 60 and 200 rows (512 leaves in all, so that levels are launched
class by class), FP64 and FP32 factors, solved without refinement.  Residuals by the
oracle: 1e-11 for FP64, 1e-4 for FP32."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def matrices(pkg, orc):
    rng = np.random.default_rng(31)
    trees = [orc.synthetic_hss(n, ls, 16, rng) for n, ls in [(16384, 128), (7680, 60), (25600, 200), (7680, 60)]]
    return [(t, pkg.HssMatrix.from_tree(t).device(), rng.standard_normal((t.size()[0], 3))) for t in trees]


@pytest.mark.parametrize("prec,bound", [("fp64", 1e-11), ("fp32", 1e-4)])
@pytest.mark.parametrize("picks", list(itertools.permutations([0, 1, 2, 3])) + [(0, 1, 3), (1, 0, 3), (1, 3, 0)])
def test_any_order(pkg, orc, matrices, picks, prec, bound):
    torch = pytest.importorskip("torch")
    from hssmatrices_gb300 import serve
    bat = serve.Batcher()
    ms = [matrices[i] for i in picks]
    facs = bat.factor([d for _t, d, _b in ms], prec)
    dB = [torch.from_numpy(np.ascontiguousarray(b.T)).cuda() for _t, _d, b in ms]
    dX = [torch.zeros_like(b) for b in dB]
    bat.solve(facs, dB, dX, [b.shape[0] for _t, _d, b in ms], [3] * len(ms), tol=-1.0)
    torch.cuda.synchronize()
    for (t, _d, b), x in zip(ms, dX):
        res = np.linalg.norm(b - orc.matmul(t, x.cpu().numpy().T)) / np.linalg.norm(b)
        assert res <= bound, t.size()
