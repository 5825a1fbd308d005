"""Launches of the panel factorization that fail (HSS_OPT_FAIL_LAUNCH: on the host,
before they reach the driver): every call that factorizes reports the error, with and
without recorded sequences, and the next one is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HSS_OPT_GRAPHS = 4


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("prec,ls,tol", [("fp64", 64, 1e-12), ("fp32", 200, 1e-8)])
@pytest.mark.parametrize("graphs", [0, 1])
def test_reported(pkg, lib, orc, prec, ls, tol, graphs):
    torch = pytest.importorskip("torch")
    L = pkg._lib
    n = 3000
    rng = np.random.default_rng(ls)
    h = orc.synthetic_hss(n, ls, 16, rng)
    b = rng.standard_normal((n, 2))
    ref = orc.ulvfactsolve(h, b)
    dev = pkg.HssMatrix.from_tree(h).device()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        dB = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
        dX = torch.zeros_like(dB)
    F = dev.ulvfactor(prec, stream=stream)

    def factsolve():
        F.factsolve_device(dB, n, 2, dX, n, tol=-1.0, stream=stream)

    def solved(bound):
        F.solve_device(dB, n, 2, dX, n, tol=-1.0, stream=stream)
        stream.synchronize()
        assert rel(dX.cpu().numpy().T, ref) <= bound

    bound = tol if prec == "fp64" else 1e-3
    calls = [lambda: dev.ulvfactor(prec, stream=stream), lambda: F.refactor(stream=stream), factsolve]
    assert lib.hss_set_option(HSS_OPT_GRAPHS, graphs) == 0
    try:
        for call in calls:
            for turn in range(4):   # with graphs: plain, recorded, replayed
                for k in (1, 2, 5):   # the first launch, a panel, one further on
                    assert lib.hss_set_option(L.HSS_OPT_FAIL_LAUNCH, k) == 0
                    try:
                        call()
                        failed = False
                    except L.HssError as e:
                        failed = True
                        assert not isinstance(e, L.HssTimeout)
                    finally:
                        lib.hss_set_option(L.HSS_OPT_FAIL_LAUNCH, 0)
                    # a replayed sequence launches nothing from the host
                    assert failed or (graphs and turn > 0 and call is not calls[0])
                call()
            F.refactor(stream=stream)
            solved(bound)
    finally:
        lib.hss_set_option(HSS_OPT_GRAPHS, 0)
    x = F.solve(b, tol=1e-10 if prec == "fp32" else 0.0)
    assert rel(x, ref) <= tol
