"""Matrices at the ends of the range in the eigensolver (csrc/eigen_dc.cu): entries
that are not finite end the call with an error on every path of the tridiagonalisation,
and the context solves the next matrix; finite ones are solved whatever their scale.

Tolerance: a backward-stable method gives eigenvalues, residual and orthogonality
within c n eps |A|_2; c = 10, the threshold of LAPACK's own test ratios."""
import numpy as np
import pytest

from imcom_b200 import EIGH_TWOSTAGE, ImcomError, Solver
from imcom_b200.api import OPT_SM_SHARE, OPT_TAIL_CTAS

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
IMCOM_ERR_EIGEN = 5


def _set(s, n):
    x = np.arange(n, dtype=float)
    s.set_inputs(x, x, np.ones(n, dtype=np.int32), x[:1], x[:1], None, None, 1.0, 1.0)


def _check(s, A):
    n = A.shape[0]
    s.load_A(np.asfortranarray(A))
    Q, L, _ = s.eigen_A()
    bound = 10 * n * EPS * np.linalg.norm(A, 2)
    assert np.abs(L - np.linalg.eigvalsh(A)[::-1]).max() <= bound
    assert np.linalg.norm((A @ Q - Q * L) / np.linalg.norm(A, 2), 2) <= 10 * n * EPS
    assert np.linalg.norm(Q.T @ Q - np.eye(n), 2) <= 10 * n * EPS


def _matrix(n):
    rng = np.random.default_rng(n)
    V = rng.standard_normal((n, n))
    return V @ V.T


@pytest.mark.parametrize("n,tail,share,two", [(2, 0, 0, False), (20, 0, 0, False), (70, 0, 0, False),
                                              (300, 8, 0, False), (300, 16, 0, False),
                                              (300, -1, 0, False), (300, 0, 3, False),
                                              (300, 0, 24, False), (2100, 0, 0, False),
                                              (300, 0, 0, True)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_finite_is_an_error(n, tail, share, two, bad):
    A = _matrix(n)
    with Solver(0) as s:
        if two:
            s.set_eigensolver(EIGH_TWOSTAGE)
        s.set_option(OPT_TAIL_CTAS, tail)
        s.set_option(OPT_SM_SHARE, share)
        _set(s, n)
        B = A.copy()
        B[n // 2, n // 3] = B[n // 3, n // 2] = bad
        s.load_A(np.asfortranarray(B))
        with pytest.raises(ImcomError) as ei:
            s.eigen_A()
        assert ei.value.status == IMCOM_ERR_EIGEN
        _check(s, A)


# A column whose squares are subnormal: its squared norm (and x^T A x against |A|) is a
# sum of n numbers, each rounded by up to 2^-1075, so the reflector and the update are
# exact to n 2^-1075 / |x|^2; 16 of these for the reflector's two sides, the update's
# terms and the two sums.
@pytest.mark.parametrize("n,split,tail", [(40, 1, 0), (40, 20, 0), (300, 1, 0), (300, 45, 0),
                                          (300, 1, -1), (300, 45, -1), (300, 45, 16),
                                          (2100, 1, 0), (2100, 40, 0)])
@pytest.mark.parametrize("tiny", [1e-153, 1e-155, 1e-156, 1e-157, 1e-158])
def test_tiny_columns(n, split, tail, tiny):
    rng = np.random.default_rng(n + split)
    A = _matrix(n) / n
    A[:split, split:] = tiny * rng.uniform(1, 2, (split, n - split))
    A[split:, :split] = A[:split, split:].T
    # |x|^2 of the first block's last column: its couplings through an orthogonal map
    norm2 = np.linalg.svd(A[:split, split:] / tiny, compute_uv=False).min() ** 2
    rel = 10 * n * EPS + 16 * n * (2.0 ** -1000 / tiny / tiny * 2.0 ** -75) / norm2
    with Solver(0) as s:
        s.set_option(OPT_TAIL_CTAS, tail)
        _set(s, n)
        s.load_A(np.asfortranarray(A))
        Q, L, _ = s.eigen_A()
    norm = np.linalg.norm(A, 2)
    assert np.abs(L - np.linalg.eigvalsh(A)[::-1]).max() <= rel * norm
    assert np.linalg.norm(A @ Q - Q * L, 2) <= rel * norm
    assert np.linalg.norm(Q.T @ Q - np.eye(n), 2) <= rel


# The reduction forms products of three entries: they leave the range at 1e-108 and
# 1e103, long before the squares of a norm do.
@pytest.mark.parametrize("n,tail,share,two", [(2, 0, 0, False), (20, 0, 0, False), (301, 0, 0, False),
                                              (300, 16, 0, False), (301, -1, 0, False),
                                              (300, 0, 3, False), (2100, 0, 0, False),
                                              (301, 0, 0, True)])
@pytest.mark.parametrize("scale", [1e-305, 1e-180, 1e-105, 1e-60, 1e-35, 1e35, 1e105, 1e180, 1e290])
def test_scaled(n, tail, share, two, scale):
    with Solver(0) as s:
        if two:
            s.set_eigensolver(EIGH_TWOSTAGE)
        s.set_option(OPT_TAIL_CTAS, tail)
        s.set_option(OPT_SM_SHARE, share)
        _set(s, n)
        _check(s, _matrix(n) * scale)


def test_powers_of_two_change_nothing():
    """Scaling is by powers of two: the same vectors to the bit, the values scaled."""
    n = 301
    A = _matrix(n)
    out = []
    with Solver(0) as s:
        _set(s, n)
        for k in (0, 99, 110, 500, -110, -500):
            s.load_A(np.asfortranarray(np.ldexp(A, k)))
            Q, L, _ = s.eigen_A()
            out.append((Q, np.ldexp(L, -k)))
    for Q, L in out[1:]:
        assert np.array_equal(Q, out[0][0])
        assert np.array_equal(L, out[0][1])


def _tridiagonal(n, mag):
    rng = np.random.default_rng(n)
    d, e = rng.uniform(1, 2, n) * mag, rng.uniform(1, 2, n - 1) * np.minimum(mag[1:], mag[:-1])
    return np.diag(d) + np.diag(e, 1) + np.diag(e, -1)


# Merges whose values are all far below the rest of the matrix (or far from 1 with all of
# it): no squares of 1 / gap that leave the range.  The matrices are tridiagonal, so the
# reduction leaves them as they are.
@pytest.mark.parametrize("n", [20, 33, 70, 71, 140, 300])
@pytest.mark.parametrize("tiny", [1e-80, 1e-100, 1e-160, 1e-300, 1e-310, 0.0])
@pytest.mark.parametrize("half", ["first", "second", "middle"])
def test_merges_of_tiny_values(n, tiny, half):
    i = np.arange(n)
    small = {"first": i < n // 2, "second": i >= n // 2, "middle": abs(i - n // 2) < n // 3}[half]
    with Solver(0) as s:
        _set(s, n)
        _check(s, _tridiagonal(n, np.where(small, tiny, 1.0)))


@pytest.mark.parametrize("n", [2, 20, 70, 300])
@pytest.mark.parametrize("scale", [1e-280, 1e-120, 1e120, 1e300])
def test_scaled_tridiagonal(n, scale):
    with Solver(0) as s:
        _set(s, n)
        _check(s, _tridiagonal(n, np.full(n, scale)))
