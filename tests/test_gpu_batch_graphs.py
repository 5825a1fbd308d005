"""Recorded launch sequences (HSS_OPT_GRAPHS) of a batcher across batches: its merged
task buffer and slot table keep their addresses, so that only the lists' keys tell a
batch of one matrix with 128-row leaves and two with 60-row leaves from one of two and
one (equal offsets, counts and largest sizes, other size classes).  Every batch's
solutions by the oracle's residual: 1e-11 for FP64 factors, 1e-4 for FP32 ones without
refinement, 1e-10 refined."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HSS_OPT_GRAPHS = 4


@pytest.fixture(scope="module")
def matrices(pkg, orc):
    rng = np.random.default_rng(31)
    # 128 leaves each: three matrices are more than two rounds of the SMs
    trees = [orc.synthetic_hss(n, ls, 16, rng) for n, ls in [(16384, 128), (7680, 60), (16384, 128), (7680, 60)]]
    return [(t, pkg.HssMatrix.from_tree(t).device(), rng.standard_normal((t.size()[0], 3))) for t in trees]


@pytest.mark.parametrize("prec,tol,bound", [("fp64", -1.0, 1e-11), ("fp32", -1.0, 1e-4), ("fp32", 1e-10, 1e-10)])
def test_batches_of_other_classes(pkg, lib, orc, matrices, prec, tol, bound):
    torch = pytest.importorskip("torch")
    from hssmatrices_gb300 import serve
    bat = serve.Batcher()
    stream = torch.cuda.Stream()
    one_two, two_one = [0, 1, 3], [0, 2, 1]
    assert lib.hss_set_option(HSS_OPT_GRAPHS, 1) == 0
    try:
        for picks in (one_two, one_two, one_two, two_one, two_one, two_one, one_two):
            ms = [matrices[i] for i in picks]
            facs = bat.factor([d for _t, d, _b in ms], prec, stream=stream)
            with torch.cuda.stream(stream):
                dB = [torch.from_numpy(np.ascontiguousarray(b.T)).cuda() for _t, _d, b in ms]
                dX = [torch.zeros_like(b) for b in dB]
            for _ in range(3):
                bat.solve(facs, dB, dX, [b.shape[0] for _t, _d, b in ms], [3] * 3, tol=tol, stream=stream)
            stream.synchronize()
            for (t, _d, b), x in zip(ms, dX):
                res = np.linalg.norm(b - orc.matmul(t, x.cpu().numpy().T)) / np.linalg.norm(b)
                assert res <= bound, (picks, t.size())
    finally:
        lib.hss_set_option(HSS_OPT_GRAPHS, 0)
