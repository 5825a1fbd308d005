"""The tensor-core sample product (``hss_sample`` with more than 2048 inner terms).

Sizes at the edges of its tiles (128 rows, chunks of 128 inner terms, column
tiles of 16 and 32) and both layouts, against exact sums.  Tolerance entrywise,
K u (|A| |X|) with u = 2^-53 and K the number of terms: the bound of an FP64 sum,
which the kernel keeps by its check (outputs for which its fixed-point digits
could do worse are summed in FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _exact(A, X):
    """A X in extended precision (at least 64 bits of mantissa)."""
    out = np.zeros((A.shape[0], X.shape[1]), dtype=np.longdouble)
    for k in range(A.shape[1]):
        out += np.outer(A[:, k].astype(np.longdouble), X[k].astype(np.longdouble))
    return out


def _host(t):
    return t.cpu().numpy().T


def _values(kind, rng, m, k):
    A = rng.standard_normal((m, k))
    if kind == "wide":                      # magnitudes over 60 decades, zeros, empty rows
        A *= 10.0 ** rng.uniform(-30, 30, size=A.shape)
        A.flat[3::7] = 0.0
        A[::5] = 0.0
    elif kind == "sparse":                  # a few entries per row
        A *= rng.random(A.shape) < 0.01
    elif kind == "digits":                  # all mantissa bits set: the largest digit sums
        A = np.where(A < 0, -1.0, 1.0) * (2.0 - 2.0 ** -52)
    elif kind == "range":                   # exponents near the ends of FP64's range, subnormals
        A *= 10.0 ** rng.choice([-310.0, -300.0, 0.0, 140.0], size=(m, 1))
    return A


@pytest.mark.parametrize("kind", ["randn", "wide", "sparse", "digits", "range"])
@pytest.mark.parametrize("m,k,r", [(1, 2049, 1), (129, 2176, 16), (300, 2300, 17), (128, 4099, 33)])
def test_sample_tc_entrywise(pkg, kind, m, k, r):
    comp = pkg.compression
    rng = np.random.default_rng(m + k + r)
    A = _values(kind, rng, m, k)
    X = rng.standard_normal((k, r))
    bound = k * U * (np.abs(A) @ np.abs(X)) + k * 5e-324
    ref = _exact(A, X)
    got = _host(comp.sample(comp.DenseDevice(A), comp._cols_to_device(X)))
    assert np.all(np.abs(got - ref) <= bound)
    got = _host(comp.sample(comp.DenseDevice(np.ascontiguousarray(A.T)), comp._cols_to_device(X), trans=True))
    assert np.all(np.abs(got - ref) <= bound)
    C0 = rng.standard_normal((m, r))
    out = comp._cols_to_device(C0)
    comp.sample(comp.DenseDevice(A), comp._cols_to_device(X), out=out, alpha=-1.0, beta=0.5)
    assert np.all(np.abs(_host(out) - (0.5 * C0 - ref)) <= 2 * bound + 4 * U * (np.abs(C0) + np.abs(ref)))


def test_sample_tc_not_finite(pkg):
    """Infinities and NaN in A or X reach exactly the outputs that an FP64 sum gives them."""
    comp = pkg.compression
    rng = np.random.default_rng(5)
    A, X = rng.standard_normal((140, 2200)), rng.standard_normal((2200, 5))
    A[3, 17], A[9, 2100], X[40, 2] = np.inf, np.nan, -np.inf
    A[20] = 0.0                              # 0 * inf
    with np.errstate(invalid="ignore"):
        ref = A @ X
    got = _host(comp.sample(comp.DenseDevice(A), comp._cols_to_device(X)))
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isposinf(got), np.isposinf(ref))
    assert np.array_equal(np.isneginf(got), np.isneginf(ref))
    f = np.isfinite(ref)
    assert np.all(np.abs(got - ref)[f] <= 2 * 2200 * U * (np.abs(A) @ np.abs(X))[f])
